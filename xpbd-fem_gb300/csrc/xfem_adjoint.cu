// Reverse-mode adjoint of the substep (sm_103a). No reference counterpart:
// the reference (jak-xyz/xpbd-fem) only steps forward. The derivative is that
// of the forward kernels' own method: predict and the velocity update
// (XPBDFEM/Geo.cpp:307-312, 342-344), the coloured Gauss-Seidel sweep of the
// coupled Neo-Hookean solve (XPBDFEM/Fem.cpp:523-553 with
// EnergyXpbdConstrainSimultaneous<2>, XPBDFEM/Xpbd.h:123-215), locks
// (XPBDFEM/Geo.cpp:318-322) and the ground projection with Coulomb friction.
//
// Tape (written by the recording forward, xfem_kernels.cu):
//   tape_v[s][v]          one 32-byte sector per vertex and substep, written
//                         by its owner: O after the advance (the substep's
//                         start position and the w its solves use) and D
//                         before it (the previous substep's swept D)
//   tape_t[s][row][lane]  each solve's input displacement (12 floats)
//   tape_fin[v]           D before the closing finalize
// Reverse order: the closing finalize, then substeps last to first, colours
// last to first; clusters of a colour share no vertex, so each updates the
// adjoint of its vertices in place (no atomics), exactly mirroring the
// forward. A cluster (one thread) walks its tets backwards from their taped
// inputs, with its vertices' adjoints in registers; the vertex owner then
// reverses the advance, as the forward did it right before its solves.
//
// Per-vertex adjoint state (AdjCtx::abar, two float4 per vertex):
//   during the run     Xb = dL/d(position O + D), Ob = dL/dO from the finish
//                      of the substep and the later ones (also across
//                      checkpoint segments, so that segmenting changes no bit)
//   end / start        dL/dX and dL/dV of the canonical state
// Per tet row: cbar += alpha0 * dL/dalpha0 + alpha1 * dL/dalpha1, which is
// -mu dL/dmu since both compliances scale as 1/mu (the host divides by -mu).
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "xfem_device.cuh"
#include "xfem_internal.h"

namespace xfem {

namespace {

__device__ __forceinline__ Vec3 vadd(Vec3 a, Vec3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ Vec3 vsub(Vec3 a, Vec3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ Vec3 vmul(Vec3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
// a + b * s
__device__ __forceinline__ Vec3 vfma(Vec3 b, float s, Vec3 a) { return {fmaf(b.x, s, a.x), fmaf(b.y, s, a.y), fmaf(b.z, s, a.z)}; }

// What one coupled solve computes, recomputed for its reverse pass from the
// tet's pre-solve state. g1_i = 2 (J - a) detQ cof_i with cof the cofactor
// rows of Ds (P1 x P2, P2 x P0, P0 x P1), so dJ/dP_i = detQ cof_i.
struct TetFw {
	Vec3 P[3], g0[4], g1[4], cof[3];
	float U0, U1, Ja, detQ, A1, l0, l1, alpha0, alpha1;
	float i00, i11, r0, r1, inv_det;  // the Cramer factors of M = [A0 A1; A1 A2]
};

__device__ __forceinline__ void tet_internals(const Mat& bp, const TetRec& r, float inv_dt2, const float4 O[4],
                                              const Vec3 D[4], TetFw& f) {
	const float q[3][3] = {{r.a.x, r.a.y, r.a.z}, {r.a.w, r.b.x, r.b.y}, {r.b.z, r.b.w, r.c.x}};
	const float QQ[3] = {r.c.y, r.c.z, r.c.w};
	const float QR[3] = {r.d.x, r.d.y, r.d.z};
	f.alpha0 = r.d.w * inv_dt2;
	f.alpha1 = f.alpha0 * bp.ratio;
#pragma unroll
	for (int i = 0; i < 3; i++)
		f.P[i] = {(O[i].x - O[3].x) + (D[i].x - D[3].x), (O[i].y - O[3].y) + (D[i].y - D[3].y),
		          (O[i].z - O[3].z) + (D[i].z - D[3].z)};
	f.U0 = deviatoric(bp, QQ, QR, f.P, f.g0);
	f.U1 = hydrostatic(q, f.P, bp.a, f.g1, &f.Ja, &f.detQ);
	f.cof[0] = cross(f.P[1], f.P[2]);
	f.cof[1] = cross(f.P[2], f.P[0]);
	f.cof[2] = cross(f.P[0], f.P[1]);
	const float w[4] = {O[0].w, O[1].w, O[2].w, O[3].w};
	const float A0 = fmaf(2.0f * f.U0, f.alpha0, wdot(w, f.g0, f.g0));
	f.A1 = wdot(w, f.g1, f.g0);
	const float A2 = fmaf(2.0f * f.U1, f.alpha1, wdot(w, f.g1, f.g1));
	f.i00 = rcp(A0);
	f.i11 = rcp(A2);
	f.r0 = f.A1 * f.i00;
	f.r1 = f.A1 * f.i11;
	f.inv_det = rcp(fmaxf(0.00000001f, fmaf(-f.r0, f.r1, 1.0f)));
	const float c0 = (-2.0f * f.U0) * f.i00, c1 = (-2.0f * f.U1) * f.i11;
	f.l0 = f.inv_det * fmaf(-f.r0, c1, c0);
	f.l1 = f.inv_det * fmaf(-c0, f.r1, c1);
}

// Reverse of one coupled solve. xb[4]: adjoint of the tet's four positions
// after the solve on entry, before it on exit. Returns
// alpha0 dL/dalpha0 + alpha1 dL/dalpha1 of this solve.
__device__ __forceinline__ float tet_reverse(const TetRec& r, const TetFw& f, const float w[4], Vec3 xb[4]) {
	const float QQ[3] = {r.c.y, r.c.z, r.c.w};
	const float QR[3] = {r.d.x, r.d.y, r.d.z};
	Vec3 gb0[4], gb1[4];
	float lb0 = 0.0f, lb1 = 0.0f;
#pragma unroll
	for (int n = 0; n < 4; n++) {
		const Vec3 y = vmul(xb[n], w[n]);
		lb0 += dot(y, f.g0[n]);
		lb1 += dot(y, f.g1[n]);
		gb0[n] = vmul(y, f.l0);
		gb1[n] = vmul(y, f.l1);
	}
	// lambda = M^-1 b with M = [A0 A1; A1 A2] symmetric: m = M^-1 lambda_bar,
	// b_bar = m, M_bar = -m lambda^T (same Cramer form as the forward)
	const float c0 = lb0 * f.i00, c1 = lb1 * f.i11;
	const float m0 = f.inv_det * fmaf(-f.r0, c1, c0);
	const float m1 = f.inv_det * fmaf(-c0, f.r1, c1);
	const float Ab0 = -m0 * f.l0, Ab2 = -m1 * f.l1, Ab1 = -fmaf(m0, f.l1, m1 * f.l0);
	// b = (-2 U0, -2 U1); A0 = sum w |g0|^2 + 2 U0 alpha0; A1 = sum w g1.g0; A2 = sum w |g1|^2 + 2 U1 alpha1
	const float Ub0 = fmaf(2.0f * f.alpha0, Ab0, -2.0f * m0);
	const float Ub1 = fmaf(2.0f * f.alpha1, Ab2, -2.0f * m1);
	const float dalpha = fmaf(f.alpha0, 2.0f * f.U0 * Ab0, f.alpha1 * (2.0f * f.U1 * Ab2));
#pragma unroll
	for (int n = 0; n < 4; n++) {
		gb0[n] = vfma(f.g0[n], 2.0f * w[n] * Ab0, vfma(f.g1[n], w[n] * Ab1, gb0[n]));
		gb1[n] = vfma(f.g1[n], 2.0f * w[n] * Ab2, vfma(f.g0[n], w[n] * Ab1, gb1[n]));
	}
	// g_3 = -(g_0 + g_1 + g_2)
#pragma unroll
	for (int i = 0; i < 3; i++) {
		gb0[i] = vsub(gb0[i], gb0[3]);
		gb1[i] = vsub(gb1[i], gb1[3]);
	}
	// deviatoric: U0 = sum QQ_i |P_i|^2 + QR . (P0.P1, P0.P2, P1.P2), g0_i = dU0/dP_i
	Vec3 Pb[3];
	Pb[0] = vfma(gb0[0], 2.0f * QQ[0], vfma(gb0[1], QR[0], vfma(gb0[2], QR[1], vmul(f.g0[0], Ub0))));
	Pb[1] = vfma(gb0[0], QR[0], vfma(gb0[1], 2.0f * QQ[1], vfma(gb0[2], QR[2], vmul(f.g0[1], Ub0))));
	Pb[2] = vfma(gb0[0], QR[1], vfma(gb0[1], QR[2], vfma(gb0[2], 2.0f * QQ[2], vmul(f.g0[2], Ub0))));
	// hydrostatic: U1 = (J - a)^2, g1_i = 2 (J - a) h_i, h_i = detQ cof_i = dJ/dP_i
	float Jb = 2.0f * f.Ja * Ub1;
	const float s2 = 2.0f * f.Ja * f.detQ;
	Vec3 cb[3];
#pragma unroll
	for (int i = 0; i < 3; i++) {
		Jb = fmaf(2.0f * f.detQ, dot(f.cof[i], gb1[i]), Jb);
		cb[i] = vmul(gb1[i], s2);
	}
#pragma unroll
	for (int i = 0; i < 3; i++) Pb[i] = vfma(f.cof[i], Jb * f.detQ, Pb[i]);
	// c = a x b: a_bar += b x c_bar, b_bar += c_bar x a
	Pb[1] = vadd(Pb[1], cross(f.P[2], cb[0]));
	Pb[2] = vadd(Pb[2], cross(cb[0], f.P[1]));
	Pb[2] = vadd(Pb[2], cross(f.P[0], cb[1]));
	Pb[0] = vadd(Pb[0], cross(cb[1], f.P[2]));
	Pb[0] = vadd(Pb[0], cross(f.P[1], cb[2]));
	Pb[1] = vadd(Pb[1], cross(cb[2], f.P[0]));
	// P_i = x_i - x_3; the identity part of x_out = x_in + w (l0 g0 + l1 g1) stays in xb
#pragma unroll
	for (int i = 0; i < 3; i++) {
		xb[i] = vadd(xb[i], Pb[i]);
		xb[3] = vsub(xb[3], Pb[i]);
	}
	return dalpha;
}

// Reverse of the finish of a substep for one vertex (finish_vertex: locks,
// then the ground projection with friction) in displacement form. Op: O of
// the substep (w before the lock), Ds: D after the sweep (flag bits in .w),
// db: dL/dD' of the finished displacement. Returns dL/dDs; adds the O part
// to ob.
__device__ __forceinline__ Vec3 finish_reverse(const BodyParams& bp, const float4& Op, const float4& Ds, Vec3 db, Vec3& ob) {
	const uint32_t bits = __float_as_uint(Ds.w);
	if (bp.lock_active && (bits & kFlagLocked)) return {0.0f, 0.0f, 0.0f};
	if (!(bp.ground && Op.w > 0.0f)) return db;
	// the forward's ground_contact, recomputed
	const Vec3 n = {bp.ground_n[0], bp.ground_n[1], bp.ground_n[2]};
	const float h = (n.x * Op.x + n.y * Op.y + n.z * Op.z) - bp.ground_d;
	const float depth = -(h + (n.x * Ds.x + n.y * Ds.y + n.z * Ds.z));
	if (!(depth > 0.0f)) return db;
	const Vec3 D1 = {Ds.x + depth * n.x, Ds.y + depth * n.y, Ds.z + depth * n.z};
	const float dn = n.x * D1.x + n.y * D1.y + n.z * D1.z;
	const Vec3 t = {D1.x - dn * n.x, D1.y - dn * n.y, D1.z - dn * n.z};
	const float lt = sqrtf(t.x * t.x + t.y * t.y + t.z * t.z);
	const float lim = bp.friction * depth;
	const bool kinetic = !(lt <= lim);
	const float sc = kinetic ? lim / lt : 1.0f;
	// D' = D1 - sc t, t = D1 - n (n . D1), D1 = Ds + depth n, depth = -(n . Op - d + n . Ds)
	Vec3 tb = vmul(db, -sc);
	float depthb = 0.0f;
	if (kinetic) {  // sc = friction depth / |t|
		const float sb = -dot(t, db);
		const float inv_lt = 1.0f / lt;
		depthb = sb * bp.friction * inv_lt;
		tb = vfma(t, -sb * sc * inv_lt * inv_lt, tb);
	}
	Vec3 D1b = vadd(db, vfma(n, -dot(n, tb), tb));
	depthb += dot(n, D1b);
	ob = vfma(n, -depthb, ob);
	return vfma(n, -depthb, D1b);
}

__device__ __forceinline__ Vec3 tip_grad(const DevCtx& C, const AdjCtx& A, uint32_t v, uint32_t run_sub) {
	const int q = __ldg(C.tip_of + v);
	if (q < 0) return {0.0f, 0.0f, 0.0f};
	return v3(__ldg(A.G + (size_t)run_sub * C.ntips + q));
}

// Tape record of vertex v at launch substep s: O after the advance, D before.
__device__ __forceinline__ const float4* tape_at(const DevCtx& C, uint32_t s, uint32_t v) {
	return C.tape_v + 2 * ((size_t)s * C.nverts + v);
}

// Where the kernels keep a vertex's adjoint state, Xb and Ob: in AdjCtx::abar,
// or spread over the shared memory of a one-cluster launch.
struct GlobalAdj {
	float4* abar;
	__device__ __forceinline__ Vec3 xb(uint32_t v) const { return v3(__ldcg(abar + 2 * (size_t)v)); }
	__device__ __forceinline__ Vec3 ob(uint32_t v) const { return v3(__ldcg(abar + 2 * (size_t)v + 1)); }
	__device__ __forceinline__ void set_xb(uint32_t v, const Vec3& a) const {
		__stcg(abar + 2 * (size_t)v, make_float4(a.x, a.y, a.z, 0.0f));
	}
	__device__ __forceinline__ void set_ob(uint32_t v, const Vec3& a) const {
		__stcg(abar + 2 * (size_t)v + 1, make_float4(a.x, a.y, a.z, 0.0f));
	}
};

struct ClusterAdj {
	ClusterVerts s;
	__device__ __forceinline__ Vec3 xb(uint32_t v) const { return v3(ClusterVerts::get(s.at(v))); }
	__device__ __forceinline__ Vec3 ob(uint32_t v) const { return v3(ClusterVerts::get(s.at(v) + 16u * s.per)); }
	__device__ __forceinline__ void set_xb(uint32_t v, const Vec3& a) const {
		ClusterVerts::put(s.at(v), make_float4(a.x, a.y, a.z, 0.0f));
	}
	__device__ __forceinline__ void set_ob(uint32_t v, const Vec3& a) const {
		ClusterVerts::put(s.at(v) + 16u * s.per, make_float4(a.x, a.y, a.z, 0.0f));
	}
};

// Reverse of the boundary between two substeps for one vertex: the finish
// of the earlier one (its start O = Op, its swept D = Ds) and the predict of
// the later one. xb: dL/d(predicted position of the later substep) with its
// solves already reversed; tip(): the loss at the end of the earlier substep, whose
// end position is the later substep's O. Leaves the earlier substep's state.
template <class AS, class Tip>
__device__ __forceinline__ void boundary_reverse(const DevCtx& C, const AS& ab, uint32_t v, const float4& Op,
                                                 const float4& Ds, Vec3 xb, Tip tip) {
	const BodyParams& bp = C.bodies[__float_as_uint(Ds.w) >> 8];
	// O of the later substep is read by its solves (through O + D), by the
	// substeps after it and by the loss
	const Vec3 os = vadd(vadd(ab.ob(v), xb), tip());
	// O = Op + D', D_pred = (D' / dt + g dt) drag dt
	const Vec3 dfin = vfma(xb, bp.drag_mul, os);
	Vec3 ob = os;
	const Vec3 dsb = finish_reverse(bp, Op, Ds, dfin, ob);
	// the earlier substep's swept position is Op + Ds
	ob = vsub(ob, dsb);
	ab.set_xb(v, dsb);
	ab.set_ob(v, ob);
}

// Reverse of advance_vertex at launch substep s for one owned vertex (xb as
// for boundary_reverse). The first substep of the run ends in the canonical
// dL/dX, dL/dV. The first substep of a later segment keeps the in-segment
// state: the previous segment's finalize reverse continues from it with the
// same arithmetic as a boundary inside a launch, so checkpointed runs give
// the full tape's results bit for bit.
// t: what it reads of the tape and the loss, loaded by the caller (owned_tape).
struct OwnedTape {
	float4 Op, Ds;  // O of the substep before (not on the launch's first), D before the advance
	Vec3 tip;       // the loss at the end of the substep before
};

__device__ __forceinline__ OwnedTape owned_tape(const DevCtx& C, const AdjCtx& A, uint32_t v, uint32_t s, bool first) {
	OwnedTape t = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), __ldcs(tape_at(C, s, v) + 1), {0.0f, 0.0f, 0.0f}};
	if (!first) {
		t.Op = __ldcg(tape_at(C, s - 1, v));
		t.tip = tip_grad(C, A, v, C.sub_base + s - 1);
	}
	return t;
}

template <class AS>
__device__ __forceinline__ void advance_reverse(const DevCtx& C, const AS& ab, uint32_t v, const OwnedTape& t, bool first,
                                                float dt, Vec3 xb) {
	if (first) {
		if (C.sub_base > 0) {
			ab.set_xb(v, xb);
			return;
		}
		// O = X, D = ((V + g dt) drag) dt
		const BodyParams& bp = C.bodies[__float_as_uint(t.Ds.w) >> 8];
		const Vec3 os = vadd(ab.ob(v), xb);
		const Vec3 vb = vmul(xb, bp.drag_mul * dt);
		ab.set_xb(v, os);
		ab.set_ob(v, vb);
		return;
	}
	boundary_reverse(C, ab, v, t.Op, t.Ds, xb, [&] { return t.tip; });
}

template <class AS>
__device__ __forceinline__ void advance_reverse(const DevCtx& C, const AdjCtx& A, const AS& ab, uint32_t v, uint32_t s,
                                                bool first, float dt, Vec3 xb) {
	if (first) {
		advance_reverse(C, ab, v, owned_tape(C, A, v, s, true), true, dt, xb);
		return;
	}
	// read where they are used: gathered first as owned_tape does, the grid form's reverse
	// of meshes that are no cubes took 1.5 to 3% longer
	boundary_reverse(C, ab, v, __ldcg(tape_at(C, s - 1, v)), __ldcs(tape_at(C, s, v) + 1), xb,
	                 [&] { return tip_grad(C, A, v, C.sub_base + s - 1); });
}

// Reverse of finalize_vertex, the launch's closing finish. For the run's last
// segment abar holds the canonical dL/dX, dL/dV at the end (plus the loss on
// the final position); for an earlier segment it holds the next segment's
// in-segment state, and the closing finish is reversed as a substep boundary.
template <class AS>
__device__ __forceinline__ void finalize_reverse(const DevCtx& C, const AdjCtx& A, const AS& ab, uint32_t v, uint32_t nsub,
                                                 float inv_dt, bool last) {
	const float4 Ds = __ldcg(C.tape_fin + v);
	const float4 Op = __ldcg(tape_at(C, nsub - 1, v));
	const uint32_t run_sub = C.sub_base + nsub - 1;
	if (!last) {
		boundary_reverse(C, ab, v, Op, Ds, ab.xb(v), [&] { return tip_grad(C, A, v, run_sub); });
		return;
	}
	const BodyParams& bp = C.bodies[__float_as_uint(Ds.w) >> 8];
	const Vec3 xcb = ab.xb(v);
	const Vec3 vcb = ab.ob(v);
	const Vec3 on = vadd(xcb, tip_grad(C, A, v, run_sub));
	// X = O + D', V = D' / dt
	const Vec3 dfin = vfma(vcb, inv_dt, on);
	Vec3 ob = on;
	const Vec3 dsb = finish_reverse(bp, Op, Ds, dfin, ob);
	ob = vsub(ob, dsb);
	ab.set_xb(v, dsb);
	ab.set_ob(v, ob);
}

// Isolated vertices: no solve touches them; one thread reverses all the
// segment's substeps of one vertex.
template <class AS>
__device__ __forceinline__ void isolated_reverse(const DevCtx& C, const AdjCtx& A, const AS& ab, uint32_t begin,
                                                 uint32_t step, uint32_t nsub, float dt) {
	for (uint32_t i = begin; i < C.nisolated; i += step) {
		const uint32_t v = __ldg(C.isolated + i);
		for (int s = (int)nsub - 1; s >= 0; s--)
			advance_reverse(C, A, ab, v, (uint32_t)s, s == 0, dt, ab.xb(v));
	}
}

// The tape's input displacement of one solve (12 floats in three float4).
__device__ __forceinline__ void load_tet_input(const DevCtx& C, uint32_t s, uint32_t row, uint32_t lane, Vec3 D[4]) {
	const float4* p = C.tape_t + ((size_t)s * C.ntrows + row) * 3 * kLanes + lane;
	const float4 a = __ldcs(p), b = __ldcs(p + kLanes), c = __ldcs(p + 2 * kLanes);
	D[0] = {a.x, a.y, a.z};
	D[1] = {a.w, b.x, b.y};
	D[2] = {b.z, b.w, c.x};
	D[3] = {c.y, c.z, c.w};
}

// One cluster (lane) of chunk block `blk`, launch substep s: reverse its
// solves last to first from their taped inputs, then the owned vertices'
// advance. CUBE: the canonical 6-tet cube with compile-time slots, all in
// registers. Records, header and vertex ids are read straight from the chunk
// block: lane-minor, so every warp load is one contiguous run.
template <bool CUBE>
__device__ __forceinline__ void cluster_reverse(const DevCtx& C, const AdjCtx& A, const float4* blk, uint32_t ntmax,
                                                uint32_t nvmax, uint32_t trow, uint32_t lane, uint32_t s, bool first,
                                                float dt, float inv_dt2) {
	constexpr uint32_t NV = CUBE ? 8u : kMaxClusterVerts;
	constexpr uint32_t NT = CUBE ? 6u : kMaxClusterTets;
	const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(blk + 4 * kLanes * ntmax);
	const uint32_t* vids = hdrs + kLanes;
	const uint32_t* slots = vids + kLanes * nvmax;
	const uint32_t hdr = __ldg(hdrs + lane);
	if ((hdr & 15u) == 0u) return;
	const uint32_t nv = CUBE ? 8u : (hdr & 15u), nt = CUBE ? 6u : ((hdr >> 4) & 15u), mask = (hdr >> 8) & 0xffu;
	const Mat mat = load_mat(C.bodies, hdr >> 16);
	uint32_t vid[NV];
	float4 O[NV];
	Vec3 xb[NV];
#pragma unroll
	for (uint32_t k = 0; k < NV; k++) {
		if (k < nv) {
			vid[k] = __ldg(vids + k * kLanes + lane);
			O[k] = __ldcg(tape_at(C, s, vid[k]));
			xb[k] = v3(__ldcg(A.abar + 2 * (size_t)vid[k]));
		}
	}
#pragma unroll
	for (int t = (int)NT - 1; t >= 0; t--) {
		if ((uint32_t)t < nt) {
			const uint32_t sl =
			    CUBE ? (uint32_t)(cube_slot(t, 0) | cube_slot(t, 1) << 4 | cube_slot(t, 2) << 8 | cube_slot(t, 3) << 12)
			         : __ldg(slots + t * kLanes + lane);
			const float4* r = blk + t * 4 * kLanes + lane;
			const TetRec tr = {__ldg(r), __ldg(r + kLanes), __ldg(r + 2 * kLanes), __ldg(r + 3 * kLanes)};
			Vec3 Din[4];
			load_tet_input(C, s, trow + t, lane, Din);
			float4 Ot[4];
			Vec3 xt[4];
			float w[4];
#pragma unroll
			for (int k = 0; k < 4; k++) {
				const uint32_t q = (sl >> (4 * k)) & 15u;
				Ot[k] = O[q];
				w[k] = O[q].w;
				xt[k] = xb[q];
			}
			TetFw f;
			tet_internals(mat, tr, inv_dt2, Ot, Din, f);
			const float dal = tet_reverse(tr, f, w, xt);
#pragma unroll
			for (int k = 0; k < 4; k++) xb[(sl >> (4 * k)) & 15u] = xt[k];
			float* cb = A.cbar + (size_t)(trow + t) * kLanes + lane;
			*cb += dal;
		}
	}
#pragma unroll
	for (uint32_t k = 0; k < NV; k++) {
		if (k < nv) {
			if (mask & (1u << k))
				advance_reverse(C, A, GlobalAdj{A.abar}, vid[k], s, first, dt, xb[k]);
			else
				__stcg(A.abar + 2 * (size_t)vid[k], make_float4(xb[k].x, xb[k].y, xb[k].z, 0.0f));
		}
	}
}

// The cube reverse with a group of 8 lanes per cluster (meshes whose colour
// passes leave most warps idle). The six solves' forward internals do not
// depend on the reverse chain, only on the tape: lanes 0-5 of the group
// recompute tet j's into shared memory side by side, then lane 0 runs the
// chain of six reverses as cluster_reverse<true> does, in the same order
// with the same arithmetic (the same results bit for bit), with one solve's
// recompute instead of six ahead of it. sh: this group's six slots; cl: the
// cluster's lane in its chunk; j: the lane's index in the group.
// One solve's slot: its forward internals and the record words its reverse
// reads (QQ in c.yzw, QR in d.xyz).
struct TetSlot {
	TetFw f;
	float4 c, d;
};

__device__ __forceinline__ void cluster_reverse_grouped(const DevCtx& C, const AdjCtx& A, const float4* blk,
                                                        uint32_t trow, uint32_t cl, uint32_t j, TetSlot* sh, uint32_t s,
                                                        bool first, float dt, float inv_dt2) {
	const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(blk + 4 * kLanes * 6);
	const uint32_t* vids = hdrs + kLanes;
	const uint32_t hdr = __ldg(hdrs + cl);
	const bool live = (hdr & 15u) != 0;
	if (live && j < 6u) {
		const Mat mat = load_mat(C.bodies, hdr >> 16);
		const float4* r = blk + j * 4 * kLanes + cl;
		const TetRec tr = {__ldg(r), __ldg(r + kLanes), __ldg(r + 2 * kLanes), __ldg(r + 3 * kLanes)};
		const uint32_t sl = (uint32_t)(cube_slot((int)j, 0) | cube_slot((int)j, 1) << 4 | cube_slot((int)j, 2) << 8 |
		                               cube_slot((int)j, 3) << 12);
		float4 Ot[4];
#pragma unroll
		for (int k = 0; k < 4; k++) Ot[k] = __ldcg(tape_at(C, s, __ldg(vids + ((sl >> (4 * k)) & 15u) * kLanes + cl)));
		Vec3 Din[4];
		load_tet_input(C, s, trow + j, cl, Din);
		tet_internals(mat, tr, inv_dt2, Ot, Din, sh[j].f);
		sh[j].c = tr.c;
		sh[j].d = tr.d;
	}
	__syncwarp();
	Vec3* xs = reinterpret_cast<Vec3*>(sh);  // after the chain: the 8 vertices' adjoints
	if (live && j == 0u) {
		float4 O[8];
		Vec3 xb[8];
#pragma unroll
		for (int k = 0; k < 8; k++) {
			const uint32_t v = __ldg(vids + k * kLanes + cl);
			O[k] = __ldcg(tape_at(C, s, v));
			xb[k] = v3(__ldcg(A.abar + 2 * (size_t)v));
		}
#pragma unroll
		for (int t = 5; t >= 0; t--) {
			const TetRec tr = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f), sh[t].c, sh[t].d};
			float w[4];
			Vec3 xt[4];
#pragma unroll
			for (int k = 0; k < 4; k++) {
				w[k] = O[cube_slot(t, k)].w;
				xt[k] = xb[cube_slot(t, k)];
			}
			const TetFw f = sh[t].f;
			const float dal = tet_reverse(tr, f, w, xt);
#pragma unroll
			for (int k = 0; k < 4; k++) xb[cube_slot(t, k)] = xt[k];
			float* cb = A.cbar + (size_t)(trow + t) * kLanes + cl;
			*cb += dal;
		}
		// the slots' reads above come first in this lane's program order
#pragma unroll
		for (int k = 0; k < 8; k++) xs[k] = xb[k];
	}
	__syncwarp();
	// lane j finishes vertex j of the cluster: its advance reverse if the
	// cluster owns it, else its adjoint
	if (live) {
		const uint32_t v = __ldg(vids + j * kLanes + cl);
		const Vec3 x = xs[j];
		if ((hdr >> (8 + j)) & 1u)
			advance_reverse(C, A, GlobalAdj{A.abar}, v, s, first, dt, x);
		else
			__stcg(A.abar + 2 * (size_t)v, make_float4(x.x, x.y, x.z, 0.0f));
	}
	__syncwarp();  // the group's slots are free for the next cluster
}

// Reverse of one recorded launch of nsub substeps (one checkpoint segment).
// Cooperative persistent grid, one warp per chunk of a colour pass; every
// colour pass ends at the bounded grid barrier, as in the forward. grouped:
// every colour pass's chunks, split in 8 parts of 4 clusters, fit the grid's
// warps at once: a warp takes one part, a group of 8 lanes per cluster
// (cluster_reverse_grouped; other chunks one lane per cluster).
__global__ void __launch_bounds__(256) k_reverse(DevCtx C, AdjCtx A, uint32_t nsub, float dt, int last, int grouped) {
	extern __shared__ __align__(16) unsigned char rsmem[];
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	const uint32_t gwarp = wib * gridDim.x + blockIdx.x, nwarps = wpb * gridDim.x;
	const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
	uint32_t target = C.bar_base;
	for (uint32_t v = gtid; v < C.nverts; v += nthreads) finalize_reverse(C, A, GlobalAdj{A.abar}, v, nsub, inv_dt, last != 0);
	bool ok = grid_sync(C, target);
	if (ok) isolated_reverse(C, A, GlobalAdj{A.abar}, gtid, nthreads, nsub, dt);
	TetSlot* gsh = reinterpret_cast<TetSlot*>(rsmem) + (size_t)wib * 24 + (lane >> 3) * 6;
	for (int s = (int)nsub - 1; s >= 0 && ok; s--) {
		for (int c = (int)C.ncolours - 1; c >= 0 && ok; c--) {
			const uint32_t cb = __ldg(C.colour_chunk_begin + c), ce = __ldg(C.colour_chunk_begin + c + 1);
			if (grouped) {
				for (uint32_t it = gwarp; it < 8u * (ce - cb); it += nwarps) {
					const uint32_t ch = cb + it / 8u, cl = (it % 8u) * 4u + (lane >> 3);
					const uint4 m = __ldg(reinterpret_cast<const uint4*>(C.chunks) + ch);
					const float4* blk = C.cblk + m.x;
					if (m.z & kShapeCube) {
						cluster_reverse_grouped(C, A, blk, m.w, cl, lane & 7u, gsh, (uint32_t)s, s == 0, dt, inv_dt2);
					} else if ((lane & 7u) == 0u) {
						cluster_reverse<false>(C, A, blk, m.z & 0xffu, (m.z >> 8) & 0xffu, m.w, cl, (uint32_t)s, s == 0,
						                       dt, inv_dt2);
					}
				}
				if (!grid_sync(C, target)) ok = false;
				continue;
			}
			for (uint32_t ch = cb + gwarp; ch < ce; ch += nwarps) {
				const uint4 m = __ldg(reinterpret_cast<const uint4*>(C.chunks) + ch);
				const float4* blk = C.cblk + m.x;
				const uint32_t ntmax = m.z & 0xffu, nvmax = (m.z >> 8) & 0xffu;
				if (m.z & kShapeCube)
					cluster_reverse<true>(C, A, blk, ntmax, nvmax, m.w, lane, (uint32_t)s, s == 0, dt, inv_dt2);
				else
					cluster_reverse<false>(C, A, blk, ntmax, nvmax, m.w, lane, (uint32_t)s, s == 0, dt, inv_dt2);
			}
			if (!grid_sync(C, target)) ok = false;
		}
	}
}

// ---- the reverse of a small all-cube handle as one thread-block cluster ---------
//
// As the forward's one-cluster form (xfem_cluster.cu): the adjoint state of
// every vertex stays in the cluster's distributed shared memory and a pass ends
// at the hardware cluster barrier. Only the chain of a cluster's six reverses
// depends on the pass before; the solves' forward internals, the inverse
// masses and what the advance reverse reads come from the tape. So a block of
// eight warps works on one chunk at a time: warp 0 runs the chain, a lane per
// cluster, while warps 1-6 recompute the internals of the block's next chunk, a
// warp per tet, and warps 1-7 load its vertices' tape; then the eight warps finish
// the chunk's eight vertices side by side. Same functions, same order: the
// gradients equal the grid form's bit for bit.
//
// 12,288 tets x 200 substeps (8 chunks per pass, 8 blocks): 11.8 ms in the grid
// form (152 blocks, 8 lanes per cluster), 6.0 ms here (10.0 before the vertex
// ids were kept in shared memory and the tape's next substep prefetched to L2,
// 7.7 while warp 7 loaded all of a chunk's vertices). A pass of 7,500 cycles: the
// chain 5,100, with the other warps' preparation of 2,500 to 4,800 beside it, the
// finish 350, the barrier 1,900.

// A cluster's tet in shared memory: TetFw and the record words its reverse
// reads, as 16 float4 per lane.
struct TetWords {
	TetFw f;
	float q[8];  // QQ, QR
};
constexpr uint32_t kTetWords4 = 16;
static_assert(sizeof(TetWords) == 16 * kTetWords4, "a tet's words are 16 float4");
constexpr uint32_t kRevColours = 16;  // colours a handle of this form has at most

// The chunk a block works on next: what its chain and finish read.
struct RevStage {
	float4 tet[6][kTetWords4][kLanes];
	float4 Op[8][kLanes], Ds[8][kLanes], tip[8][kLanes];
	float w[8][kLanes];
};

struct RevShared {
	RevStage st[2];
	float4 xb[8][kLanes];
};

// A chunk of the block's, kept for the launch: headers, vertex ids, first tet
// row and the sums of -mu dL/dmu.
struct RevChunk {
	uint32_t hdr[kLanes], vid[8][kLanes];
	float cbar[6][kLanes];
	uint32_t off16, trow, pad[2];
};

// The cube's tets turn around its diagonal (solve_cube): in reverse, odd
// tets (0, 3, N, P), then even ones (0, N, P, 3), the ring moved back by two
// places per turn.
__device__ __forceinline__ void reverse_cube(const RevStage& S, uint32_t lane, Vec3 xb[8], float* cbar) {
	Vec3 r[6] = {xb[6], xb[7], xb[2], xb[1], xb[4], xb[5]};
	float rw[6] = {S.w[6][lane], S.w[7][lane], S.w[2][lane], S.w[1][lane], S.w[4][lane], S.w[5][lane]};
	const float w0 = S.w[0][lane], w3 = S.w[3][lane];
	Vec3 x0 = xb[0], x3 = xb[3];
	auto one = [&](int t, const float w[4], Vec3 x[4]) {
		TetWords tw;
		float4 words[kTetWords4];
#pragma unroll
		for (uint32_t k = 0; k < kTetWords4; k++) words[k] = S.tet[t][k][lane];
		memcpy(&tw, words, sizeof(tw));
		const TetRec tr = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f),
		                   make_float4(0.0f, tw.q[0], tw.q[1], tw.q[2]), make_float4(tw.q[3], tw.q[4], tw.q[5], 0.0f)};
		cbar[t * kLanes] += tet_reverse(tr, tw.f, w, x);
	};
#pragma unroll 1
	for (int t = 4; t >= 0; t -= 2) {
		{
			const float w[4] = {w0, w3, rw[2], rw[1]};
			Vec3 x[4] = {x0, x3, r[2], r[1]};
			one(t + 1, w, x);
			x0 = x[0], x3 = x[1], r[2] = x[2], r[1] = x[3];
		}
		{
			const float w[4] = {w0, rw[1], rw[0], w3};
			Vec3 x[4] = {x0, r[1], r[0], x3};
			one(t, w, x);
			x0 = x[0], r[1] = x[1], r[0] = x[2], x3 = x[3];
		}
		const Vec3 a = r[4], b = r[5];
		const float wa = rw[4], wb = rw[5];
#pragma unroll
		for (int k = 5; k >= 2; k--) r[k] = r[k - 2], rw[k] = rw[k - 2];
		r[0] = a, r[1] = b, rw[0] = wa, rw[1] = wb;
	}
	xb[0] = x0, xb[3] = x3;
	// three turns back by two: the places of the first turn again
	xb[6] = r[0], xb[7] = r[1], xb[2] = r[2], xb[1] = r[3], xb[4] = r[4], xb[5] = r[5];
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Tet j of chunk R: its internals at launch substep s, and the same tape entry of
// the substep before to L2.
__device__ __forceinline__ void reverse_prepare_tet(const DevCtx& C, RevStage& S, const RevChunk& R, uint32_t s, uint32_t j,
                                                    uint32_t lane, uint32_t hdr, float inv_dt2) {
	const Mat mat = load_mat(C.bodies, hdr >> 16);
	const float4* r = C.cblk + R.off16 + j * 4 * kLanes + lane;
	const TetRec tr = {__ldg(r), __ldg(r + kLanes), __ldg(r + 2 * kLanes), __ldg(r + 3 * kLanes)};
	const uint32_t sl = (uint32_t)(cube_slot((int)j, 0) | cube_slot((int)j, 1) << 4 | cube_slot((int)j, 2) << 8 |
	                               cube_slot((int)j, 3) << 12);
	float4 Ot[4];
#pragma unroll
	for (int k = 0; k < 4; k++) Ot[k] = __ldcg(tape_at(C, s, R.vid[(sl >> (4 * k)) & 15u][lane]));
	Vec3 Din[4];
	load_tet_input(C, s, R.trow + j, lane, Din);
	if (s > 0u) {
		const float4* p = C.tape_t + ((size_t)(s - 1u) * C.ntrows + R.trow + j) * 3 * kLanes + lane;
		prefetch_l2(p);
		prefetch_l2(p + kLanes);
		prefetch_l2(p + 2 * kLanes);
	}
	TetWords tw;
	tet_internals(mat, tr, inv_dt2, Ot, Din, tw.f);
	const float q[8] = {tr.c.y, tr.c.z, tr.c.w, tr.d.x, tr.d.y, tr.d.z, 0.0f, 0.0f};
#pragma unroll
	for (int k = 0; k < 8; k++) tw.q[k] = q[k];
	float4 words[kTetWords4];
	memcpy(words, &tw, sizeof(tw));
#pragma unroll
	for (uint32_t k = 0; k < kTetWords4; k++) S.tet[j][k][lane] = words[k];
}

// Warp `wib` (1-7) of the block prepares chunk R at launch substep s, and has
// the same entries of the substep before it brought to L2 (the tape of a long
// run comes from HBM).
__device__ __forceinline__ void reverse_prepare(const DevCtx& C, const AdjCtx& A, RevStage& S, const RevChunk& R,
                                                uint32_t s, bool first, uint32_t wib, uint32_t lane, float inv_dt2) {
	const uint32_t hdr = R.hdr[lane];
	if ((hdr & 15u) == 0u) return;
	// What the finish reads of vertex wib - 1 (warp 7: also of vertex 7) is loaded
	// ahead of the tet. All eight by warp 7 took it 6,700 cycles, 1,800 longer than
	// the chain.
	float vw[2];
	OwnedTape own[2];
#pragma unroll
	for (uint32_t i = 0; i < 2u; i++) {
		const uint32_t k = wib - 1u + i;
		if (i == 1u && wib != 7u) break;
		const uint32_t v = R.vid[k][lane];
		vw[i] = __ldcg(&tape_at(C, s, v)->w);
		if ((hdr >> (8 + k)) & 1u) own[i] = owned_tape(C, A, v, s, first);
		if (s > 0u) prefetch_l2(tape_at(C, s - 1u, v));
	}
	if (wib < 7u) reverse_prepare_tet(C, S, R, s, wib - 1u, lane, hdr, inv_dt2);
#pragma unroll
	for (uint32_t i = 0; i < 2u; i++) {
		const uint32_t k = wib - 1u + i;
		if (i == 1u && wib != 7u) break;
		S.w[k][lane] = vw[i];
		if ((hdr >> (8 + k)) & 1u) {
			S.Op[k][lane] = own[i].Op;
			S.Ds[k][lane] = own[i].Ds;
			S.tip[k][lane] = make_float4(own[i].tip.x, own[i].tip.y, own[i].tip.z, 0.0f);
		}
	}
}

__global__ void __launch_bounds__(256, 1) k_reverse_cluster(DevCtx C, AdjCtx A, uint32_t nsub, float dt, int last,
                                                            uint32_t rounds) {
	extern __shared__ __align__(128) unsigned char rcmem[];
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
	const uint32_t G = gridDim.x, rank = blockIdx.x;
	RevShared& S = *reinterpret_cast<RevShared*>(rcmem);
	float4* sv = reinterpret_cast<float4*>(rcmem + sizeof(RevShared));
	const uint32_t per = cluster_verts(C.nverts, G);
	RevChunk* chunks = reinterpret_cast<RevChunk*>(sv + 2 * (size_t)per);  // [colour][round]
	const ClusterAdj ab = {ClusterVerts(smem_u32(sv), per)};
	const uint32_t v0 = min(rank * per, C.nverts), v1 = min(v0 + per, C.nverts);
	for (uint32_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
		sv[v - v0] = __ldcg(A.abar + 2 * (size_t)v);
		sv[per + (v - v0)] = __ldcg(A.abar + 2 * (size_t)v + 1);
		finalize_reverse(C, A, ab, v, nsub, inv_dt, last != 0);
	}
	// the block's chunks of each colour, in rounds: [first, end)
	__shared__ uint32_t s_first[kRevColours], s_end[kRevColours];
	if (threadIdx.x < C.ncolours) {
		const uint32_t cb = __ldg(C.colour_chunk_begin + threadIdx.x), n = __ldg(C.colour_chunk_begin + threadIdx.x + 1) - cb;
		s_first[threadIdx.x] = cb + n * rank / G;
		s_end[threadIdx.x] = cb + n * (rank + 1u) / G;
	}
	__syncthreads();
	for (uint32_t c = 0; c < C.ncolours; c++)
		for (uint32_t k = 0; s_first[c] + k < s_end[c]; k++) {
			RevChunk& R = chunks[c * rounds + k];
			const uint4 m = __ldg(reinterpret_cast<const uint4*>(C.chunks) + s_first[c] + k);
			const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(C.cblk + m.x + 4 * kLanes * 6);
			for (uint32_t i = threadIdx.x; i < 9u * kLanes; i += blockDim.x) (&R.hdr[0])[i] = __ldg(hdrs + i);
			for (uint32_t i = threadIdx.x; i < 6u * kLanes; i += blockDim.x) (&R.cbar[0][0])[i] = A.cbar[(size_t)m.w * kLanes + i];
			if (threadIdx.x == 0) R.off16 = m.x, R.trow = m.w;
		}
	cluster_barrier();
	isolated_reverse(C, A, ab, rank * blockDim.x + threadIdx.x, G * blockDim.x, nsub, dt);

	// the block's next chunk after (s, c, k), -1 when there is none
	auto next_of = [&](int& s, int& c, uint32_t& k) {
		if (s_first[c] + k + 1u < s_end[c]) {
			k++;
			return true;
		}
		for (;;) {
			if (--c < 0) {
				c = (int)C.ncolours - 1;
				if (--s < 0) return false;
			}
			if (s_first[c] < s_end[c]) {
				k = 0;
				return true;
			}
		}
	};
	// the first chunk of the launch
	int ns = (int)nsub - 1, nc = (int)C.ncolours - 1;
	uint32_t nk = 0, it = 0;
	bool more = s_first[nc] < s_end[nc] || next_of(ns, nc, nk);
	if (more && wib > 0)
		reverse_prepare(C, A, S.st[0], chunks[(uint32_t)nc * rounds + nk], (uint32_t)ns, ns == 0, wib, lane, inv_dt2);
	for (int s = (int)nsub - 1; s >= 0; s--) {
		for (int c = (int)C.ncolours - 1; c >= 0; c--) {
			const uint32_t cf = s_first[c], n = s_end[c] - cf;
			for (uint32_t k = 0; k < n; k++, it++) {
				__syncthreads();  // the chunk is prepared, the last one finished
				RevStage& st = S.st[it & 1u];
				more = next_of(ns, nc, nk);
				RevChunk& R = chunks[(uint32_t)c * rounds + k];
				const uint32_t hdr = R.hdr[lane];
				const bool live = (hdr & 15u) != 0u;
				if (wib == 0) {
					if (live) {
						Vec3 xb[8];
#pragma unroll
						for (uint32_t j = 0; j < 8u; j++) xb[j] = ab.xb(R.vid[j][lane]);
						reverse_cube(st, lane, xb, &R.cbar[0][lane]);
#pragma unroll
						for (uint32_t j = 0; j < 8u; j++) S.xb[j][lane] = make_float4(xb[j].x, xb[j].y, xb[j].z, 0.0f);
					}
				} else if (more) {
					reverse_prepare(C, A, S.st[(it + 1u) & 1u], chunks[(uint32_t)nc * rounds + nk], (uint32_t)ns, ns == 0, wib, lane,
					                inv_dt2);
				}
				__syncthreads();
				// warp j finishes vertex j of each cluster: its advance reverse if
				// the cluster owns it, else its adjoint
				if (live) {
					const uint32_t v = R.vid[wib][lane];
					const Vec3 x = v3(S.xb[wib][lane]);
					if ((hdr >> (8 + wib)) & 1u)
						advance_reverse(C, ab, v, OwnedTape{st.Op[wib][lane], st.Ds[wib][lane], v3(st.tip[wib][lane])}, s == 0, dt, x);
					else
						ab.set_xb(v, x);
				}
			}
			cluster_barrier();
		}
	}
	for (uint32_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
		__stcg(A.abar + 2 * (size_t)v, sv[v - v0]);
		__stcg(A.abar + 2 * (size_t)v + 1, sv[per + (v - v0)]);
	}
	for (uint32_t c = 0; c < C.ncolours; c++)
		for (uint32_t k = 0; s_first[c] + k < s_end[c]; k++) {
			const RevChunk& R = chunks[c * rounds + k];
			for (uint32_t i = threadIdx.x; i < 6u * kLanes; i += blockDim.x)
				A.cbar[(size_t)R.trow * kLanes + i] = (&R.cbar[0][0])[i];
		}
}

// Blocks of the one-cluster reverse, 0 when the handle does not take it: all
// clusters whole cubes, at most 16 colours and at most two chunks of a colour per
// block. The grid form takes any number of chunks up to one per SM in about the
// same time, the cluster one round of its blocks after the other. Measured, 50
// substeps, cluster and grid: 16 chunks of a colour (one round) 1,476 and 2,992 us,
// 18 and 32 (two) 2,614 and 3,026, 2,560 and 3,101; 34 and 40 (three) 3,253 and
// 3,049, 3,726 and 3,209.
cudaError_t reverse_cluster_blocks(const DevCtx& C, uint32_t max_colour_chunks, uint32_t* blocks, uint32_t* rounds,
                                   size_t* smem) {
	*blocks = 0;
	if (C.vs_off != C.warp_smem || C.ncolours == 0 || C.ncolours > kRevColours || max_colour_chunks == 0) return cudaSuccess;
	uint32_t G = 1;
	while (G < 16u && G < max_colour_chunks) G *= 2;
	*rounds = (max_colour_chunks + G - 1) / G;
	if (*rounds > 2u) return cudaSuccess;
	int dev = 0, optin = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
	const void* f = (const void*)k_reverse_cluster;
	cudaFuncAttributes fa{};
	if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f);
	if (e != cudaSuccess) return e;
	*smem = sizeof(RevShared) + 32u * (size_t)cluster_verts(C.nverts, G) + sizeof(RevChunk) * (size_t)C.ncolours * *rounds;
	if (*smem + fa.sharedSizeBytes > (size_t)optin) return cudaSuccess;
	e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
	cudaLaunchAttribute at{};
	at.id = cudaLaunchAttributeClusterDimension;
	at.val.clusterDim.x = G;
	at.val.clusterDim.y = at.val.clusterDim.z = 1;
	cudaLaunchConfig_t lc{};
	lc.gridDim = dim3(G);
	lc.blockDim = dim3(256);
	lc.dynamicSmemBytes = *smem;
	lc.attrs = &at;
	lc.numAttrs = 1;
	int n = 0;
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, f, &lc);
	if (e == cudaSuccess && n > 0) *blocks = G;
	return e;
}

}  // namespace

int configure_adjoint_kernels(int, uint32_t) { return 0; }

int launch_reverse(const DevCtx& ctx, const AdjCtx& adj, int block, uint32_t, uint32_t max_colour_chunks, uint32_t nsub,
                   float dt, bool last, void* stream) {
	if (nsub == 0) return 0;
	cudaStream_t st = (cudaStream_t)stream;
	const char* form = getenv("XFEM_REVERSE_FORM");
	// the hooks that make grid-barrier waits run out or wrap need that barrier
	if (!form && !ctx.wait_miss && !ctx.bar_base) {
		uint32_t G = 0, rounds = 0;
		size_t bytes = 0;
		const cudaError_t ec = reverse_cluster_blocks(ctx, max_colour_chunks, &G, &rounds, &bytes);
		if (ec != cudaSuccess) return (int)ec;
		if (G) {
			cudaLaunchAttribute at{};
			at.id = cudaLaunchAttributeClusterDimension;
			at.val.clusterDim.x = G;
			at.val.clusterDim.y = at.val.clusterDim.z = 1;
			cudaLaunchConfig_t lc{};
			lc.gridDim = dim3(G);
			lc.blockDim = dim3(256);
			lc.dynamicSmemBytes = bytes;
			lc.stream = st;
			lc.attrs = &at;
			lc.numAttrs = 1;
			DevCtx c = ctx;
			AdjCtx a = adj;
			int lastv = last ? 1 : 0;
			void* args[] = {&c, &a, &nsub, &dt, &lastv, &rounds};
			note_launch(XFEM_FORM_CLUSTER, G, 256, 1);
			return (int)cudaLaunchKernelExC(&lc, (const void*)k_reverse_cluster, args);
		}
	}
	int dev = 0, sms = 0, per_sm = 0;
	// six forward-internal slots per 8-lane group, 4 groups per warp
	const size_t smem = (size_t)(block / 32) * 24 * sizeof(TetSlot);
	cudaError_t e = cudaFuncSetAttribute((const void*)k_reverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e == cudaSuccess) e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_reverse, block, smem);
	if (e != cudaSuccess) return (int)e;
	if (per_sm <= 0) return (int)cudaErrorInvalidConfiguration;
	// the whole co-resident grid, as the forward: chunk i of a colour goes to
	// block i % grid, so a colour pass with fewer chunks than warps still
	// spreads one chunk per SM (a pass lasts as long as its slowest chunk)
	const uint32_t blocks = (uint32_t)(per_sm * sms);
	e = reset_barrier(ctx, st);
	if (e != cudaSuccess) return (int)e;
	DevCtx c = ctx;
	AdjCtx a = adj;
	int lastv = last ? 1 : 0;
	// the grouped form when one round of the grid's warps takes every part of
	// the largest colour pass
	int grouped = (uint64_t)max_colour_chunks * 8u <= (uint64_t)blocks * (uint32_t)(block / 32) ? 1 : 0;
	if (form) grouped = form[0] == 'g' ? 1 : form[0] == 'l' ? 0 : grouped;
	void* args[] = {&c, &a, &nsub, &dt, &lastv, &grouped};
	note_launch(XFEM_FORM_GRID, blocks, (uint32_t)block, grouped ? 8 : 1);
	return (int)cudaLaunchCooperativeKernel((const void*)k_reverse, dim3(blocks), dim3(block), args, smem, st);
}

}  // namespace xfem
