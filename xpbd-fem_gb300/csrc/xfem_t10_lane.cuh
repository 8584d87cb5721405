// A T10 by one lane (sm_103a): the solves of the four-lane form
// (xfem_t10_elem.cuh) in the same order, bit for bit. For meshes and solves that
// run faster that way (t10_lanes, xfem_api.cpp). Included by one kernel's file
// each: ptxas 13.0 crashes on one out-of-line device function called from two
// kernels of one file.
#pragma once

#include "xfem_t10_elem.cuh"

namespace xfem {

namespace {

namespace t10e {

// (J - a)^2 over the 4 points (weight 1/4 each) into U, g
__device__ __forceinline__ void q_hydro(const DevCtx& C, const float Qi[3][3], const Vec3 P[9], float a, float& U,
                                        Vec3 g[10]) {
#pragma unroll 1
	for (int p = 0; p < 4; p++) {
		float F[3][3], A[3][3], G[3][3];
		q_def_grad(C, Qi, p, P, F);
		const float Ja = adj_det(F, A) - a;
		U = fmaf(0.25f * Ja, Ja, U);
		const float s = 0.5f * Ja;
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) G[c][r] = A[c][r] * s;
		q_apply(C, G, Qi, p, g);
	}
}

// The Pixar models (mu / 2 = 1): Full and Reduced on the 4 points, Selective
// the hydrostatic term on them and I1 prefactored
__device__ __forceinline__ float q_pixar(const DevCtx& C, const QRec& R, const BodyParams& bp, uint32_t e,
                                         const float Qi[3][3], const Vec3 P[9], Vec3 g[10]) {
	const float a = __ldg(&bp.a), hw = __ldg(&bp.hw);
	float U = 0.0f;
	zeron<10>(g);
	if (e != 2u) {
#pragma unroll 1
		for (int p = 0; p < 4; p++) {
			float F[3][3], A[3][3], G[3][3];
			q_def_grad(C, Qi, p, P, F);
			const float Ja = adj_det(F, A) - a;
			U = fmaf(0.25f, fmaf(hw * Ja, Ja, trace_xtx(F)), U);
			const float s2 = 0.5f * hw * Ja;
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) G[c][r] = fmaf(F[r][c], 0.5f, A[c][r] * s2);
			q_apply(C, G, Qi, p, g);
		}
		rootn<10>(g);
		return U;
	}
	q_hydro(C, Qi, P, a, U, g);
	U *= hw;
#pragma unroll
	for (int n = 0; n < 9; n++) g[n] = {g[n].x * hw, g[n].y * hw, g[n].z * hw};
	rootn<10>(g);
	Vec3 gi[10];
	U += q_pref_i1(R, P, gi);
#pragma unroll
	for (int n = 0; n < 10; n++) g[n] = {g[n].x + gi[n].x, g[n].y + gi[n].y, g[n].z + gi[n].z};
	return U;
}

// The deviatoric term on the 4 points (Mixed, YeohSkin, YeohSkinSel) with
// the hydrostatic term in the same loop when `coupled`; returns U0 before
// the clamp
__device__ __forceinline__ float q_dev_full(const DevCtx& C, const BodyParams& bp, uint32_t e, const float Qi[3][3],
                                            const Vec3 P[9], bool coupled, Vec3 g0[10], float& U1, Vec3 g1[10]) {
	const float a = __ldg(&bp.a);
	const float C0 = __ldg(&bp.yeoh[0]), C1 = __ldg(&bp.yeoh[1]), C2 = __ldg(&bp.yeoh[2]);
	float U0 = 0.0f;
#pragma unroll 1
	for (int p = 0; p < 4; p++) {
		float F[3][3], A[3][3], G[3][3];
		q_def_grad(C, Qi, p, P, F);
		const float J = adj_det(F, A);
		const float I1 = trace_xtx(F);
		float s;
		if (e == 3u) {
			U0 = fmaf(0.25f, I1, U0);
			s = 0.5f;
		} else {
			const float IM = I1 - 3.0f;
			U0 = fmaf(0.25f, IM * fmaf(IM, fmaf(IM, C2, C1), C0), U0);
			s = 0.5f * fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
		}
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) G[c][r] = F[r][c] * s;
		q_apply(C, G, Qi, p, g0);
		if (coupled) {
			const float Ja = J - a;
			U1 = fmaf(0.25f * Ja, Ja, U1);
			const float s1 = 0.5f * Ja;
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) G[c][r] = A[c][r] * s1;
			q_apply(C, G, Qi, p, g1);
		}
	}
	return U0;
}

// One T10 of a pass by one lane (the kinds of ElemPass; kRayleigh with the Rayleigh
// ratio rd).
template <int KIND>
__device__ __noinline__ void q_pass(const DevCtx& C, uint32_t i, float inv_dt, float inv_dt2, float rd) {
	uint32_t dv[10];
	q_load(C, i, dv);
	float4 O[10], D[10];
#pragma unroll
	for (int n = 0; n < 10; n++) ld_vertex(C.vert + 2 * (size_t)dv[n], O[n], D[n]);
	const BodyParams& bp = C.bodies[__float_as_uint(D[0].w) >> 8];
	const uint32_t e = __ldg(&bp.energy);
	if (KIND != kVolume && (e == 11u || e == 12u)) return;  // SolveElementCube acts on quads and hexes only
	const QRec R{C.el_rec, C.nel, i};
	float w[10];
#pragma unroll
	for (int n = 0; n < 10; n++) w[n] = O[n].w;
	float Qi[3][3];
#pragma unroll
	for (int c = 0; c < 3; c++)
#pragma unroll
		for (int r = 0; r < 3; r++) Qi[c][r] = R(kQQi + 3 * c + r);
	const float vol = R(kQVol);
	const uint32_t type = __ldg(&bp.rayleigh_type);
	const float damp = KIND == kSolve && type < 2u ? __ldg(&bp.damping) : 0.0f;
	const bool limit = type == 1u;
	const bool sim = __ldg(&bp.simultaneous) != 0u;
	Vec3 P[9], g0[10], g1[10];
	q_rel(O, D, KIND == kRayleigh, P);
	if (KIND == kVolume) {
		float U = 0.0f;
		zeron<10>(g0);
		q_hydro(C, Qi, P, 1.0f, U, g0);
		rootn<10>(g0);
		const float alpha = __ldg(&bp.compliance) * vol * inv_dt2;
		moven<10>(w, (-2.0f * U) / fmaf(2.0f * U, alpha, wdotn<10>(w, g0, g0)), g0, D);
	} else if (e <= 2u) {
		const float U = q_pixar(C, R, bp, e, Qi, P, g0);
		const float comp = __ldg(&bp.compliance) / vol;
		if (KIND == kRayleigh)
			moven<10>(w, -gdotn<10>(g0, D) / fmaf(2.0f * U, comp * inv_dt / rd, wdotn<10>(w, g0, g0)), g0, D);
		else
			moven<10>(w, lambda1n<10>(U, g0, w, D, comp * inv_dt2, comp, damp, limit, inv_dt), g0, D);
	} else {
		const float a = __ldg(&bp.a);
		const float comp0 = __ldg(&bp.inv_mu) / vol, comp1 = __ldg(&bp.inv_lambda) / vol;
		const float alpha0 = comp0 * inv_dt2, alpha1 = comp1 * inv_dt2;
		const bool coupled = KIND == kRayleigh || sim;
		const bool full = full_quadrature(e);
		float U0, U1 = 0.0f;
		zeron<10>(g0);
		zeron<10>(g1);
		if (full) {
			U0 = fmaxf(0.0001f, q_dev_full(C, bp, e, Qi, P, coupled && e != 6u, g0, U1, g1));
			rootn<10>(g0);
		} else {
			U0 = q_pref_i1(R, P, g0);
			if (e == 7u) {
				const float C0 = __ldg(&bp.yeoh[0]), C1 = __ldg(&bp.yeoh[1]), C2 = __ldg(&bp.yeoh[2]);
				const float IM = U0 - 3.0f;
				U0 = fmaxf(0.0001f, IM * fmaf(IM, fmaf(IM, C2, C1), C0));
				const float gs = fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
#pragma unroll
				for (int n = 0; n < 10; n++) g0[n] = {g0[n].x * gs, g0[n].y * gs, g0[n].z * gs};
			}
		}
		if (coupled) {
			if (!full || e == 6u) q_hydro(C, Qi, P, a, U1, g1);
			rootn<10>(g1);
			if (KIND == kRayleigh) {
				if (sim) {
					const float b0 = -gdotn<10>(g0, D), b1 = -gdotn<10>(g1, D);
					float l0, l1;
					cramer(fmaf(2.0f * U0, comp0 * inv_dt / rd, wdotn<10>(w, g0, g0)), wdotn<10>(w, g0, g1),
					       fmaf(2.0f * U1, comp1 * inv_dt / rd, wdotn<10>(w, g1, g1)), b0, b1, l0, l1);
#pragma unroll
					for (int n = 0; n < 10; n++) {
						const float s0 = w[n] * l0, s1 = w[n] * l1;
						D[n].x = fmaf(s1, g1[n].x, fmaf(s0, g0[n].x, D[n].x));
						D[n].y = fmaf(s1, g1[n].y, fmaf(s0, g0[n].y, D[n].y));
						D[n].z = fmaf(s1, g1[n].z, fmaf(s0, g0[n].z, D[n].z));
					}
				} else {
					moven<10>(w, -gdotn<10>(g0, D) / fmaf(2.0f * U0, comp0 * inv_dt / rd, wdotn<10>(w, g0, g0)), g0, D);
					moven<10>(w, -gdotn<10>(g1, D) / fmaf(2.0f * U1, comp1 * inv_dt / rd, wdotn<10>(w, g1, g1)), g1, D);
				}
			} else {
				float l0, l1;
				lambda2n<10>(U0, U1, g0, g1, w, D, alpha0, alpha1, comp0, comp1, damp, limit, inv_dt, l0, l1);
#pragma unroll
				for (int n = 0; n < 10; n++) {
					const float s0 = w[n] * l0, s1 = w[n] * l1;
					D[n].x = fmaf(s1, g1[n].x, fmaf(s0, g0[n].x, D[n].x));
					D[n].y = fmaf(s1, g1[n].y, fmaf(s0, g0[n].y, D[n].y));
					D[n].z = fmaf(s1, g1[n].z, fmaf(s0, g0[n].z, D[n].z));
				}
			}
		} else {
			// serial: deviatoric, refresh P, hydrostatic
			moven<10>(w, lambda1n<10>(U0, g0, w, D, alpha0, comp0, damp, limit, inv_dt), g0, D);
			q_rel(O, D, false, P);
			q_hydro(C, Qi, P, a, U1, g1);
			rootn<10>(g1);
			moven<10>(w, lambda1n<10>(U1, g1, w, D, alpha1, comp1, damp, limit, inv_dt), g1, D);
		}
	}
#pragma unroll
	for (int n = 0; n < 10; n++) st_vertex(C.vert + 2 * (size_t)dv[n], O[n], D[n]);
}

// A lane per T10: meshes whose colours fill the GPU that way.
struct T10Lane {
	static constexpr int kLanes = 1, kPbdLanes = 1;
	static constexpr int kBlock = 256, kMinBlocks = 1;
	static constexpr uint32_t kVid4 = 3;
	static constexpr size_t smem() { return 0; }
	__device__ static void init(const DevCtx&) {}
	template <int KIND>
	__device__ static void pass(const DevCtx& C, uint32_t i, uint32_t, bool, float inv_dt, float inv_dt2, float rd) {
		q_pass<KIND>(C, i, inv_dt, inv_dt2, rd);
	}
	__device__ static void pbd(const DevCtx& C, uint32_t i, float coeff) { q_pbd(C, i, coeff); }
};

}  // namespace t10e

}  // namespace

}  // namespace xfem
