// Quadratic-tet element code of libxfem.so (sm_103a), shared by the T10
// mode (xfem_t10.cu) and meshes mixing T10s and H27s (xfem_qmixed.cu): GeoQuadratic3d on a tet mesh
// (XPBDFEM/Geo.cpp:836-1053). Every tet gets a node on each edge
// (Connectivity3d's edge numbering); SolveElement on ElementParamsQuadraticTet
// (XPBDFEM/Fem.cpp:871-893: SolveElementPixar :361-433 and SolveElementMixed
// :437-564 with Nodes = 10 and the 4-point rule, PointsLo = PointsHi = 4; the
// cube models leave a tet alone), SolveVolumeOnly (:840-867), DampElement
// (:910-928) and PbdDamp (XPBDFEM/Xpbd.h:306-346), in the element kernel of
// xfem_elements.cuh with four lanes of a warp per T10 or one (t10_lanes, xfem_api.cpp).
//
// Records: 14 float4 per T10 as a structure of arrays (float4 k of element i
// at el_rec[k * nel + i]): Qi column-major, volume, surface area, the
// prefactored QQ[9] and QR[36]. The map from the corners is linear, so one
// Qi serves all four points; their shape-function gradients come from a
// 120-float table (el_tab).
#pragma once

#include "xfem_elements.cuh"

namespace xfem {

namespace {

namespace t10e {

constexpr int kQQi = 0, kQVol = 9, kQArea = 10, kQQQ = 11, kQQR = 20;

struct QRec {
	const float4* base;
	uint32_t n, i;
	__device__ __forceinline__ float operator()(int j) const {
		return __ldg(reinterpret_cast<const float*>(base + (size_t)(j >> 2) * n + i) + (j & 3));
	}
};

__device__ __forceinline__ float g4(const DevCtx& C, int p, int n, int k) { return __ldg(C.el_tab + (p * 10 + n) * 3 + k); }

// F = Qi MatMul(dN[0..8], P) at point p (XPBDFEM/Fem.cpp:311-316)
__device__ __forceinline__ void q_def_grad(const DevCtx& C, const float Qi[3][3], int p, const Vec3 P[9], float F[3][3]) {
	float Dm[3][3];
#pragma unroll
	for (int r = 0; r < 3; r++) {
		float x = 0.0f, y = 0.0f, z = 0.0f;
#pragma unroll
		for (int n = 0; n < 9; n++) {
			const float d = g4(C, p, n, r);
			x = fmaf(d, P[n].x, x);
			y = fmaf(d, P[n].y, y);
			z = fmaf(d, P[n].z, z);
		}
		Dm[0][r] = x;
		Dm[1][r] = y;
		Dm[2][r] = z;
	}
#pragma unroll
	for (int c = 0; c < 3; c++)
#pragma unroll
		for (int r = 0; r < 3; r++) F[c][r] = fmaf(Qi[0][r], Dm[c][0], fmaf(Qi[1][r], Dm[c][1], Qi[2][r] * Dm[c][2]));
}

// ApplyEnergyGradient with the constant Qi: g[n] += (G Qi) dN[n], n < 9
__device__ __forceinline__ void q_apply(const DevCtx& C, const float G[3][3], const float Qi[3][3], int p, Vec3 g[10]) {
	float M[3][3];
#pragma unroll
	for (int j = 0; j < 3; j++)
#pragma unroll
		for (int r = 0; r < 3; r++) M[j][r] = fmaf(G[0][r], Qi[j][0], fmaf(G[1][r], Qi[j][1], G[2][r] * Qi[j][2]));
#pragma unroll
	for (int n = 0; n < 9; n++) {
		const float d0 = g4(C, p, n, 0), d1 = g4(C, p, n, 1), d2 = g4(C, p, n, 2);
		g[n].x += fmaf(M[0][0], d0, fmaf(M[1][0], d1, M[2][0] * d2));
		g[n].y += fmaf(M[0][1], d0, fmaf(M[1][1], d1, M[2][1] * d2));
		g[n].z += fmaf(M[0][2], d0, fmaf(M[1][2], d1, M[2][2] * d2));
	}
}

__device__ __forceinline__ float trace_xtx(const float F[3][3]) {
	return fmaf(F[0][0], F[0][0], fmaf(F[0][1], F[0][1], F[0][2] * F[0][2])) +
	       fmaf(F[1][0], F[1][0], fmaf(F[1][1], F[1][1], F[1][2] * F[1][2])) +
	       fmaf(F[2][0], F[2][0], fmaf(F[2][1], F[2][1], F[2][2] * F[2][2]));
}

// I1 prefactored over the nine edge vectors (XPBDFEM/Fem.cpp:163-192),
// root gradient included
__device__ __forceinline__ float q_pref_i1(const QRec& R, const Vec3 P[9], Vec3 g[10]) {
	float U = 0.0f;
#pragma unroll
	for (int i = 0; i < 9; i++) {
		const float qq = R(kQQQ + i);
		U = fmaf(qq, dot(P[i], P[i]), U);
		const float d = 2.0f * qq;
		g[i] = {d * P[i].x, d * P[i].y, d * P[i].z};
	}
	int k = 0;
#pragma unroll
	for (int i = 0; i < 9; i++)
#pragma unroll
		for (int j = i + 1; j < 9; j++, k++) {
			const float qr = R(kQQR + k);
			U = fmaf(qr, dot(P[i], P[j]), U);
			g[i] = {fmaf(qr, P[j].x, g[i].x), fmaf(qr, P[j].y, g[i].y), fmaf(qr, P[j].z, g[i].z)};
			g[j] = {fmaf(qr, P[i].x, g[j].x), fmaf(qr, P[i].y, g[j].y), fmaf(qr, P[i].z, g[j].z)};
		}
	g[9] = {0.0f, 0.0f, 0.0f};
	rootn<10>(g);
	return U;
}

__device__ __forceinline__ void q_load(const DevCtx& C, uint32_t i, uint32_t dv[10]) {
	const uint4 a = __ldg(C.el_vid + 3 * (size_t)i), b = __ldg(C.el_vid + 3 * (size_t)i + 1),
	            c = __ldg(C.el_vid + 3 * (size_t)i + 2);
	dv[0] = a.x, dv[1] = a.y, dv[2] = a.z, dv[3] = a.w, dv[4] = b.x, dv[5] = b.y, dv[6] = b.z, dv[7] = b.w;
	dv[8] = c.x, dv[9] = c.y;
}

__device__ __forceinline__ void q_rel(const float4 O[10], const float4 D[10], bool vmode, Vec3 P[9]) {
#pragma unroll
	for (int i = 0; i < 9; i++)
		P[i] = vmode ? Vec3{O[i].x - O[9].x, O[i].y - O[9].y, O[i].z - O[9].z}
		             : Vec3{(O[i].x - O[9].x) + (D[i].x - D[9].x), (O[i].y - O[9].y) + (D[i].y - D[9].y),
		                    (O[i].z - O[9].z) + (D[i].z - D[9].z)};
}

// ---- one T10 by four lanes ----------------------------------------------------
//
// A colour pass of a mesh has a few thousand T10s, so a thread that takes a
// whole one leaves most of the SM idle for the length of its chain (3,500
// instructions, 255 registers). Here four lanes of a warp share a T10, eight
// T10s a warp: lane l forms the deformation gradient at point l, and owns
// nodes l, l + 4 and l + 8 (their loads, gradients, products and updates). What
// passes between the lanes goes through the warp's shared memory; every sum
// runs over the points, pairs and nodes in the one-lane order on every lane, so
// the results do not depend on the split.
//
// 230,400 T10s (31 colours of up to 10,080), 20 substeps: 4,202 us with a lane
// per T10, 3,515 us with four and the next eight fetched ahead. Twelve warps a
// block: with eight, a colour of 10,000 needs a second round of a few warps
// (3,855 us); with sixteen the registers spill (3,914 us). Solves and sizes that
// run faster with a lane per T10, whose work per element is less, keep one
// (xfem_t10_lane.cuh; four_lane_share in xfem_api.cpp, at most one round of these
// warps: 14,592 T10s of a colour on 152 SMs).

// A warp's shared memory. rec: the records, element-major (60 floats apart:
// eight elements' 16-byte reads fall in different banks); the others
// [row][element].
struct QuadScratch {
	float rec[8][60];
	uint32_t vid[8][12];  // the T10s' vertex ids
	uint32_t have;        // the warp's first T10 whose record and ids are here or on their way
	uint32_t pad[3];
	float4 P[10][8];       // node offsets from node 9 (row 9: unused by the solves; D rows with damping)
	float4 M0[12][8], M1[12][8];  // per point three rows: the energy gradient mapped back (9 values)
	float4 g0[10][8], g1[10][8];  // the nodes' gradients
	float4 dots[10][8];    // per node: g0.g0, g1.g0, g1.g1, w
};
constexpr int kQuadWarps = (int)kT10QuadWarps;
struct QuadShared {
	float4 tab[40];  // shape-function gradients, [point][node]
	QuadScratch w[kQuadWarps];
};

__device__ __forceinline__ QuadShared& quad_shared() {
	extern __shared__ __align__(128) unsigned char qsmem[];
	return *reinterpret_cast<QuadShared*>(qsmem);
}

// The calling lane's share of one T10.
struct Quad {
	QuadScratch& S;
	const float4* tab;
	uint32_t lane, e, l;  // e: element slot of the warp, l: lane of the element
	float4 O[3], D[3];    // nodes l, l + 4, l + 8 (the last: l < 2)
	uint32_t dv[3];
	float Qi[3][3];

	__device__ __forceinline__ Quad(QuadShared& q)
	    : S(q.w[threadIdx.x >> 5]), tab(q.tab), lane(threadIdx.x & 31u), e(lane >> 2), l(lane & 3u) {}

	__device__ __forceinline__ bool has(int k) const { return k < 2 || l < 2u; }
	__device__ __forceinline__ float rec(int j) const { return S.rec[e][j]; }
	__device__ __forceinline__ float group(float x, uint32_t src) const {
		return __shfl_sync(0xffffffffu, x, (lane & ~3u) + src);
	}
	static __device__ __forceinline__ Vec3 xyz(const float4& a) { return {a.x, a.y, a.z}; }
	static __device__ __forceinline__ float4 f4(const Vec3& a) { return make_float4(a.x, a.y, a.z, 0.0f); }

	// Starts the copy of the records and vertex ids of the warp's eight
	// elements from i0 on (up to `last`): asynchronous 16-byte copies.
	__device__ __forceinline__ void fetch(const DevCtx& C, uint32_t i0, uint32_t last) {
		__syncwarp();  // every lane is done with the last elements' copies
		auto copy = [](void* dst, const void* from) {
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(from) : "memory");
		};
#pragma unroll
		for (uint32_t t = 0; t < 4u; t++) {
			const uint32_t x = lane + 32u * t, k = x >> 3, el = x & 7u;
			if (k < 14u) copy(&S.rec[el][4 * k], C.el_rec + (size_t)k * C.nel + min(i0 + el, last));
		}
		if (lane < 24u) {
			const uint32_t el = lane / 3u, k = lane - 3u * el;
			copy(&S.vid[el][4 * k], C.el_vid + 3 * (size_t)min(i0 + el, last) + k);
		}
		if (lane == 0) S.have = i0;
		__syncwarp();
	}

	// The warp's eight elements from i0 on (up to `last`), this lane's nodes.
	__device__ __forceinline__ void load(const DevCtx& C, uint32_t i0, uint32_t last) {
		if (S.have != i0) {
			asm volatile("cp.async.wait_all;" ::: "memory");  // a fetch that is not used after all
			fetch(C, i0, last);
		}
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncwarp();
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (has(k)) {
				dv[k] = S.vid[e][l + 4 * k];
				ld_vertex(C.vert + 2 * (size_t)dv[k], O[k], D[k]);
			} else {
				dv[k] = 0;
				O[k] = D[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			}
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) Qi[c][r] = rec(kQQi + 3 * c + r);
	}

	// The nodes' offsets from node 9 (lane 1's third).
	__device__ __forceinline__ void share_rel(bool vmode) {
		const float ox = group(O[2].x, 1), oy = group(O[2].y, 1), oz = group(O[2].z, 1);
		const float dx = group(D[2].x, 1), dy = group(D[2].y, 1), dz = group(D[2].z, 1);
		__syncwarp();
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (k < 2 || l == 0u)
				S.P[l + 4 * k][e] = vmode ? make_float4(O[k].x - ox, O[k].y - oy, O[k].z - oz, 0.0f)
				                          : make_float4((O[k].x - ox) + (D[k].x - dx), (O[k].y - oy) + (D[k].y - dy),
				                                        (O[k].z - oz) + (D[k].z - dz), 0.0f);
		__syncwarp();
	}

	__device__ __forceinline__ void def_grad(float F[3][3]) const {
		float Dm[3][3] = {};
#pragma unroll
		for (int n = 0; n < 9; n++) {
			const float4 d = tab[l * 10u + n], p = S.P[n][e];
			Dm[0][0] = fmaf(d.x, p.x, Dm[0][0]), Dm[1][0] = fmaf(d.x, p.y, Dm[1][0]), Dm[2][0] = fmaf(d.x, p.z, Dm[2][0]);
			Dm[0][1] = fmaf(d.y, p.x, Dm[0][1]), Dm[1][1] = fmaf(d.y, p.y, Dm[1][1]), Dm[2][1] = fmaf(d.y, p.z, Dm[2][1]);
			Dm[0][2] = fmaf(d.z, p.x, Dm[0][2]), Dm[1][2] = fmaf(d.z, p.y, Dm[1][2]), Dm[2][2] = fmaf(d.z, p.z, Dm[2][2]);
		}
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) F[c][r] = fmaf(Qi[0][r], Dm[c][0], fmaf(Qi[1][r], Dm[c][1], Qi[2][r] * Dm[c][2]));
	}

	// (G Qi) of this lane's point
	__device__ __forceinline__ void put(float4 (*M)[8], const float G[3][3]) {
		float m[9];
#pragma unroll
		for (int j = 0; j < 3; j++)
#pragma unroll
			for (int r = 0; r < 3; r++) m[3 * j + r] = fmaf(G[0][r], Qi[j][0], fmaf(G[1][r], Qi[j][1], G[2][r] * Qi[j][2]));
		M[3 * l][e] = make_float4(m[0], m[1], m[2], 0.0f);
		M[3 * l + 1][e] = make_float4(m[3], m[4], m[5], 0.0f);
		M[3 * l + 2][e] = make_float4(m[6], m[7], m[8], 0.0f);
	}

	// g[n] += (G Qi) dN[n] over the points, for this lane's nodes below 9
	__device__ __forceinline__ void gather(const float4 (*M)[8], Vec3 g[3]) const {
#pragma unroll
		for (int k = 0; k < 3; k++) g[k] = {0.0f, 0.0f, 0.0f};
#pragma unroll
		for (int p = 0; p < 4; p++) {
			const float4 a = M[3 * p][e], b = M[3 * p + 1][e], c = M[3 * p + 2][e];
#pragma unroll
			for (int k = 0; k < 3; k++)
				if (k < 2 || l == 0u) {
					const float4 d = tab[p * 10u + l + 4 * k];
					g[k].x += fmaf(a.x, d.x, fmaf(b.x, d.y, c.x * d.z));
					g[k].y += fmaf(a.y, d.x, fmaf(b.y, d.y, c.y * d.z));
					g[k].z += fmaf(a.z, d.x, fmaf(b.z, d.y, c.z * d.z));
				}
		}
	}

	// Leaves the gradients of nodes 0-8 in G's rows; node 9 takes minus
	// their sum.
	__device__ __forceinline__ void root(float4 (*G)[8], Vec3 g[3]) {
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (k < 2 || l == 0u) G[l + 4 * k][e] = f4(g[k]);
		__syncwarp();
		if (l == 1u) {
			Vec3 s = {0.0f, 0.0f, 0.0f};
#pragma unroll
			for (int n = 0; n < 9; n++) {
				const float4 a = G[n][e];
				s = {s.x + a.x, s.y + a.y, s.z + a.z};
			}
			g[2] = {0.0f - s.x, 0.0f - s.y, 0.0f - s.z};
		}
	}

	// The same for two gradients at once.
	__device__ __forceinline__ void root2(Vec3 g0[3], Vec3 g1[3]) {
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (k < 2 || l == 0u) S.g0[l + 4 * k][e] = f4(g0[k]), S.g1[l + 4 * k][e] = f4(g1[k]);
		__syncwarp();
		if (l == 1u) {
			Vec3 s = {0.0f, 0.0f, 0.0f}, t = {0.0f, 0.0f, 0.0f};
#pragma unroll
			for (int n = 0; n < 9; n++) {
				const float4 a = S.g0[n][e], b = S.g1[n][e];
				s = {s.x + a.x, s.y + a.y, s.z + a.z};
				t = {t.x + b.x, t.y + b.y, t.z + b.z};
			}
			g0[2] = {0.0f - s.x, 0.0f - s.y, 0.0f - s.z};
			g1[2] = {0.0f - t.x, 0.0f - t.y, 0.0f - t.z};
		}
	}

	// (J - a)^2 over the points into M1; returns U (every lane).
	__device__ __forceinline__ float hydro(float a) {
		float F[3][3], A[3][3], G[3][3];
		def_grad(F);
		const float Ja = adj_det(F, A) - a;
		const float s = 0.5f * Ja;
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) G[c][r] = A[c][r] * s;
		put(S.M1, G);
		return sum_sq(Ja);
	}
	__device__ __forceinline__ float sum_sq(float Ja) const {
		float U = 0.0f;
#pragma unroll
		for (int p = 0; p < 4; p++) {
			const float x = group(Ja, p);
			U = fmaf(0.25f * x, x, U);
		}
		return U;
	}
	__device__ __forceinline__ float sum4(float v) const {
		float U = 0.0f;
#pragma unroll
		for (int p = 0; p < 4; p++) U = fmaf(0.25f, group(v, p), U);
		return U;
	}

	// The full Pixar energy (Pixar, PixarReduced; mu / 2 = 1) into M0, or the
	// deviatoric term (Mixed, YeohSkin, YeohSkinSel) into M0 with the hydrostatic
	// one into M1 (U1 when `coupled`), a lane per point.
	__device__ __forceinline__ float pixar_full(float a, float hw) {
		float F[3][3], A[3][3], G[3][3];
		def_grad(F);
		const float Ja = adj_det(F, A) - a;
		const float v = fmaf(hw * Ja, Ja, trace_xtx(F));
		const float s2 = 0.5f * hw * Ja;
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) G[c][r] = fmaf(F[r][c], 0.5f, A[c][r] * s2);
		put(S.M0, G);
		return sum4(v);
	}
	__device__ __forceinline__ float dev_full(const BodyParams& bp, uint32_t en, bool coupled, float& U1) {
		const float a = __ldg(&bp.a);
		const float C0 = __ldg(&bp.yeoh[0]), C1 = __ldg(&bp.yeoh[1]), C2 = __ldg(&bp.yeoh[2]);
		float F[3][3], A[3][3], G[3][3];
		def_grad(F);
		const float J = adj_det(F, A);
		const float I1 = trace_xtx(F);
		float v, s;
		if (en == 3u) {
			v = I1;
			s = 0.5f;
		} else {
			const float IM = I1 - 3.0f;
			v = IM * fmaf(IM, fmaf(IM, C2, C1), C0);
			s = 0.5f * fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
		}
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) G[c][r] = F[r][c] * s;
		put(S.M0, G);
		const float Ja = J - a;
		const float s1 = 0.5f * Ja;
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) G[c][r] = A[c][r] * s1;
		put(S.M1, G);
		if (coupled) U1 = sum_sq(Ja);
		return sum4(v);
	}

	// I1 prefactored: U on every lane, this lane's nodes' gradients below 9.
	// Pair (i, j), i < j, has coefficient i (17 - i) / 2 + j - i - 1 of QR.
	__device__ __forceinline__ float pref_i1(Vec3 g[3]) const {
		Vec3 P[9];
#pragma unroll
		for (int n = 0; n < 9; n++) P[n] = xyz(S.P[n][e]);
		float U = 0.0f;
#pragma unroll
		for (int i = 0; i < 9; i++) U = fmaf(rec(kQQQ + i), dot(P[i], P[i]), U);
		int q = 0;
#pragma unroll
		for (int i = 0; i < 9; i++)
#pragma unroll
			for (int j = i + 1; j < 9; j++, q++) U = fmaf(rec(kQQR + q), dot(P[i], P[j]), U);
		// no branches: the pair's place is selected, and m = n adds 0 P_n (node 9
		// of lane 1 and the lanes without a third node compute a row no one reads)
#pragma unroll
		for (int k = 0; k < 3; k++) {
			const int n = k == 2 ? 8 : (int)l + 4 * k;
			const float d = 2.0f * S.rec[e][kQQQ + n];
			const Vec3 Pn = xyz(S.P[n][e]);
			g[k] = {d * Pn.x, d * Pn.y, d * Pn.z};
			const int below = kQQR + n - 1;                       // + m (17 - m) / 2 - m: pairs (m, n)
			const int above = kQQR + n * (17 - n) / 2 - n - 1;  // + m: pairs (n, m)
#pragma unroll
			for (int m = 0; m < 9; m++) {
				if (k == 2 && m == 8) continue;
				const float q = S.rec[e][k == 2 || m < n ? below + (m * (17 - m) / 2 - m) : above + m];
				const float qr = k < 2 && m == n ? 0.0f : q;
				g[k] = {fmaf(qr, P[m].x, g[k].x), fmaf(qr, P[m].y, g[k].y), fmaf(qr, P[m].z, g[k].z)};
			}
		}
		return U;
	}

	// The weighted products over the nodes, in node order.
	__device__ __forceinline__ void wdots(const Vec3 g0[3], const Vec3 g1[3], float& s00, float& s10, float& s11) {
		__syncwarp();
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (has(k)) S.dots[l + 4 * k][e] = make_float4(dot(g0[k], g0[k]), dot(g1[k], g0[k]), dot(g1[k], g1[k]), O[k].w);
		__syncwarp();
		s00 = s10 = s11 = 1.0e-22f;
#pragma unroll
		for (int n = 0; n < 10; n++) {
			const float4 d = S.dots[n][e];
			s00 = fmaf(d.w, d.x, s00);
			s10 = fmaf(d.w, d.y, s10);
			s11 = fmaf(d.w, d.z, s11);
		}
	}

	// sum g.D over the nodes in node order (damping only): D left in P's rows
	// (the callers form P again before they read it).
	__device__ __forceinline__ float gdot(float4 (*G)[8], const Vec3 g[3]) {
		__syncwarp();
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (has(k)) {
				G[l + 4 * k][e] = f4(g[k]);
				S.P[l + 4 * k][e] = D[k];
			}
		__syncwarp();
		float s = 0.0f;
#pragma unroll
		for (int n = 0; n < 10; n++) {
			const float4 a = G[n][e], d = S.P[n][e];
			s = fmaf(a.x, d.x, fmaf(a.y, d.y, fmaf(a.z, d.z, s)));
		}
		return s;
	}

	__device__ __forceinline__ void move(float lam, const Vec3 g[3]) {
#pragma unroll
		for (int k = 0; k < 3; k++) {
			const float s = O[k].w * lam;
			D[k].x = fmaf(s, g[k].x, D[k].x);
			D[k].y = fmaf(s, g[k].y, D[k].y);
			D[k].z = fmaf(s, g[k].z, D[k].z);
		}
	}
	__device__ __forceinline__ void move2(float l0, const Vec3 g0[3], float l1, const Vec3 g1[3]) {
#pragma unroll
		for (int k = 0; k < 3; k++) {
			const float s0 = O[k].w * l0, s1 = O[k].w * l1;
			D[k].x = fmaf(s1, g1[k].x, fmaf(s0, g0[k].x, D[k].x));
			D[k].y = fmaf(s1, g1[k].y, fmaf(s0, g0[k].y, D[k].y));
			D[k].z = fmaf(s1, g1[k].z, fmaf(s0, g0[k].z, D[k].z));
		}
	}
};

// The solve of a T10 whose deviatoric term is prefactored, coupled and without
// in-solve damping (MixedSel, YeohSkinFast and ids above 12), which is most of
// them: quad_general's branch for it, straight.
__device__ __forceinline__ void quad_coupled(Quad& Q, const BodyParams& bp, uint32_t en, float inv_dt2, float inv_dt) {
	Vec3 g0[3], g1[3];
	float s00, s10, s11;
	const float U1 = Q.hydro(__ldg(&bp.a));
	float U0 = Q.pref_i1(g0);
	__syncwarp();
	Q.gather(Q.S.M1, g1);
	Q.root2(g0, g1);
	if (en == 7u) {
		const float C0 = __ldg(&bp.yeoh[0]), C1 = __ldg(&bp.yeoh[1]), C2 = __ldg(&bp.yeoh[2]);
		const float IM = U0 - 3.0f;
		U0 = fmaxf(0.0001f, IM * fmaf(IM, fmaf(IM, C2, C1), C0));
		const float gs = fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
#pragma unroll
		for (int k = 0; k < 3; k++) g0[k] = {g0[k].x * gs, g0[k].y * gs, g0[k].z * gs};
	}
	Q.wdots(g0, g1, s00, s10, s11);
	const float vol = Q.rec(kQVol);
	const float comp0 = __ldg(&bp.inv_mu) / vol, comp1 = __ldg(&bp.inv_lambda) / vol;
	float l0, l1;
	lambda2_of(U0, U1, s00, s10, s11, 0.0f, 0.0f, comp0 * inv_dt2, comp1 * inv_dt2, comp0, comp1, 0.0f, false, inv_dt, l0, l1);
	Q.move2(l0, g0, l1, g1);
}

// Every other energy, damping and pass kind (the kinds of ElemPass; kRayleigh
// with the Rayleigh ratio rd), on the loaded Q. Branches on the energy are per
// group, and groups meet at warp barriers in them: the warp's elements all run
// the branch of any of them, and each keeps its own.
template <int KIND>
__device__ __noinline__ void quad_general(Quad& Q, const BodyParams& bp, uint32_t en, float inv_dt, float inv_dt2, float rd) {
	const float vol = Q.rec(kQVol);
	const uint32_t type = __ldg(&bp.rayleigh_type);
	const float damp = KIND == kSolve && type < 2u ? __ldg(&bp.damping) : 0.0f;
	const bool limit = type == 1u;
	const bool sim = __ldg(&bp.simultaneous) != 0u;
	auto any = [](bool x) { return __any_sync(0xffffffffu, x); };
	const bool damped = any(damp > 0.0f);
	Vec3 g0[3], g1[3];
	float s00, s10, s11;
	if (KIND == kVolume) {
		const float U = Q.hydro(1.0f);
		__syncwarp();
		Q.gather(Q.S.M1, g0);
		Q.root(Q.S.g0, g0);
		Q.wdots(g0, g0, s00, s10, s11);
		const float alpha = __ldg(&bp.compliance) * vol * inv_dt2;
		Q.move((-2.0f * U) / fmaf(2.0f * U, alpha, s00), g0);
	} else {
		const bool pixar = en <= 2u;
		if (any(pixar)) {
			const float4 D0 = Q.D[0], D1 = Q.D[1], D2 = Q.D[2];
			// the energy on the points and the selective one each where some group has
			// it (230,400 T10s of the former, 20 substeps: 5,118 us with both, 3,637 so)
			const float a = __ldg(&bp.a), hw = __ldg(&bp.hw);
			float U = 0.0f;
#pragma unroll
			for (int k = 0; k < 3; k++) g0[k] = {0.0f, 0.0f, 0.0f};
			if (any(en < 2u)) {
				U = Q.pixar_full(a, hw);
				__syncwarp();
				Q.gather(Q.S.M0, g0);
				Q.root(Q.S.g0, g0);
			}
			if (any(en == 2u)) {
				const float Uh = Q.hydro(a) * hw;
				__syncwarp();
				Q.gather(Q.S.M1, g1);
#pragma unroll
				for (int k = 0; k < 3; k++) g1[k] = {g1[k].x * hw, g1[k].y * hw, g1[k].z * hw};
				Q.root(Q.S.g1, g1);
				Vec3 gi[3];
				const float Up = Q.pref_i1(gi);
				__syncwarp();
				Q.root(Q.S.dots, gi);
				if (en == 2u) {
					U = Uh + Up;
#pragma unroll
					for (int k = 0; k < 3; k++) g0[k] = {g1[k].x + gi[k].x, g1[k].y + gi[k].y, g1[k].z + gi[k].z};
				}
			}
			const float comp = __ldg(&bp.compliance) / vol;
			Q.wdots(g0, g0, s00, s10, s11);
			float gV = 0.0f;
			if (KIND == kRayleigh || damped) gV = Q.gdot(Q.S.g0, g0);
			if (KIND == kRayleigh)
				Q.move(-gV / fmaf(2.0f * U, comp * inv_dt / rd, s00), g0);
			else
				Q.move(lambda1_of(U, s00, damp > 0.0f ? gV : 0.0f, comp * inv_dt2, comp, damp, limit, inv_dt), g0);
			if (!pixar) Q.D[0] = D0, Q.D[1] = D1, Q.D[2] = D2;
			if (any(!pixar)) Q.share_rel(KIND == kRayleigh);
		}
		if (any(!pixar)) {
			const float4 D0 = Q.D[0], D1 = Q.D[1], D2 = Q.D[2];
			const float a = __ldg(&bp.a);
			const float comp0 = __ldg(&bp.inv_mu) / vol, comp1 = __ldg(&bp.inv_lambda) / vol;
			const float alpha0 = comp0 * inv_dt2, alpha1 = comp1 * inv_dt2;
			const bool coupled = KIND == kRayleigh || sim;
			const bool full = full_quadrature(en);
			float U0 = 0.0f, U1 = 0.0f;
			if (any(full)) {
				// groups of other energies read their own rows again below
				const float Uf = Q.dev_full(bp, en, true, U1);
				__syncwarp();
				Q.gather(Q.S.M0, g0);
				Q.root(Q.S.g0, g0);
				U0 = fmaxf(0.0001f, Uf);
			}
			if (any(!full)) {
				Vec3 gp[3];
				float Up = Q.pref_i1(gp);
				__syncwarp();
				Q.root(Q.S.dots, gp);
				if (en == 7u) {
					const float C0 = __ldg(&bp.yeoh[0]), C1 = __ldg(&bp.yeoh[1]), C2 = __ldg(&bp.yeoh[2]);
					const float IM = Up - 3.0f;
					Up = fmaxf(0.0001f, IM * fmaf(IM, fmaf(IM, C2, C1), C0));
					const float gs = fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
#pragma unroll
					for (int k = 0; k < 3; k++) gp[k] = {gp[k].x * gs, gp[k].y * gs, gp[k].z * gs};
				}
				if (!full) {
					U0 = Up;
#pragma unroll
					for (int k = 0; k < 3; k++) g0[k] = gp[k];
				}
			}
			if (any(coupled)) {
				if (any(!full)) {
					// the same terms as dev_full's M1 where a group has them already
					U1 = Q.hydro(a);
					__syncwarp();
				}
				Q.gather(Q.S.M1, g1);
				Q.root(Q.S.g1, g1);
				Q.wdots(g0, g1, s00, s10, s11);
				float gV0 = 0.0f, gV1 = 0.0f;
				if (KIND == kRayleigh || damped) {
					gV0 = Q.gdot(Q.S.g0, g0);
					gV1 = Q.gdot(Q.S.g1, g1);
				}
				if (KIND == kRayleigh) {
					if (sim) {
						float l0, l1;
						cramer(fmaf(2.0f * U0, comp0 * inv_dt / rd, s00), s10, fmaf(2.0f * U1, comp1 * inv_dt / rd, s11), -gV0, -gV1,
						       l0, l1);
						Q.move2(l0, g0, l1, g1);
					}
					if (any(!sim)) {
						// one constraint after the other: the second sees the first's move
						if (!sim) Q.move(-gV0 / fmaf(2.0f * U0, comp0 * inv_dt / rd, s00), g0);
						const float gV = Q.gdot(Q.S.g1, g1);
						if (!sim) Q.move(-gV / fmaf(2.0f * U1, comp1 * inv_dt / rd, s11), g1);
					}
				} else if (coupled) {
					float l0, l1;
					lambda2_of(U0, U1, s00, s10, s11, damp > 0.0f ? gV0 : 0.0f, damp > 0.0f ? gV1 : 0.0f, alpha0, alpha1, comp0,
					           comp1, damp, limit, inv_dt, l0, l1);
					Q.move2(l0, g0, l1, g1);
				}
			}
			if (KIND != kRayleigh && any(!coupled)) {
				// serial: deviatoric, refresh P, hydrostatic
				Q.wdots(g0, g0, s00, s10, s11);
				float gV = 0.0f;
				if (damped) gV = Q.gdot(Q.S.g0, g0);
				if (!coupled) Q.move(lambda1_of(U0, s00, damp > 0.0f ? gV : 0.0f, alpha0, comp0, damp, limit, inv_dt), g0);
				Q.share_rel(false);
				U1 = Q.hydro(a);
				__syncwarp();
				Q.gather(Q.S.M1, g1);
				Q.root(Q.S.g1, g1);
				Q.wdots(g1, g1, s00, s10, s11);
				if (damped) gV = Q.gdot(Q.S.g1, g1);
				if (!coupled) Q.move(lambda1_of(U1, s00, damp > 0.0f ? gV : 0.0f, alpha1, comp1, damp, limit, inv_dt), g1);
			}
			if (pixar) Q.D[0] = D0, Q.D[1] = D1, Q.D[2] = D2;
		}
	}
}

// Eight T10s of a pass by the calling warp: the elements from i0 on, i0 + e of
// the lane's group (a group past `last`, or not `live`, takes part without
// storing); next: the warp's next call's i0 (kNoElem: none), up to next_last.
template <int KIND>
__device__ __noinline__ void quad_pass(const DevCtx& C, uint32_t i0, uint32_t last, bool live, uint32_t next,
                                       uint32_t next_last, float inv_dt, float inv_dt2, float rd) {
	Quad Q(quad_shared());
	Q.load(C, i0, last);
	const BodyParams& bp = C.bodies[__float_as_uint(Q.group(Q.D[0].w, 0)) >> 8];
	const uint32_t en = __ldg(&bp.energy);
	live = live && (KIND == kVolume || (en != 11u && en != 12u));  // SolveElementCube acts on quads and hexes only
	Q.share_rel(KIND == kRayleigh);
	bool other = KIND != kSolve;
	if (KIND == kSolve)
		other = __any_sync(0xffffffffu, en <= 2u || full_quadrature(en) || __ldg(&bp.simultaneous) == 0u ||
		                                    (__ldg(&bp.rayleigh_type) < 2u && __ldg(&bp.damping) > 0.0f));
	if (other) {
		Quad G = Q;  // a copy: Q itself stays in registers
		quad_general<KIND>(G, bp, en, inv_dt, inv_dt2, rd);
#pragma unroll
		for (int k = 0; k < 3; k++) Q.D[k] = G.D[k];
	} else {
		quad_coupled(Q, bp, en, inv_dt2, inv_dt);
	}
	if (next != kNoElem) Q.fetch(C, next, next_last);
	if (live) {
#pragma unroll
		for (int k = 0; k < 3; k++)
			if (Q.has(k)) st_vertex(C.vert + 2 * (size_t)Q.dv[k], Q.O[k], Q.D[k]);
	}
}

__device__ __noinline__ void q_pbd(const DevCtx& C, uint32_t i, float coeff) {
	uint32_t dv[10];
	q_load(C, i, dv);
	pbd_nodes<10>(C, dv, fminf(1.0f, coeff / QRec{C.el_rec, C.nel, i}(kQArea)));
}

struct T10Elem {
	static constexpr int kLanes = 4, kPbdLanes = 1;
	static constexpr int kBlock = 32 * kQuadWarps, kMinBlocks = 1;
	static constexpr uint32_t kVid4 = 3;
	static constexpr size_t smem() { return sizeof(QuadShared); }
	__device__ static void init(const DevCtx& C) {
		for (uint32_t k = threadIdx.x; k < 40u; k += blockDim.x)
			quad_shared().tab[k] = make_float4(__ldg(C.el_tab + 3 * k), __ldg(C.el_tab + 3 * k + 1), __ldg(C.el_tab + 3 * k + 2), 0.0f);
		if ((threadIdx.x & 31u) == 0u) quad_shared().w[threadIdx.x >> 5].have = kNoElem;
		__syncthreads();
	}
	template <int KIND>
	__device__ static void pass(const DevCtx& C, uint32_t i0, uint32_t last, bool live, float inv_dt, float inv_dt2, float rd,
	                            uint32_t next = kNoElem, uint32_t next_last = 0) {
		quad_pass<KIND>(C, i0, last, live, next, next_last, inv_dt, inv_dt2, rd);
	}
	__device__ static void pbd(const DevCtx& C, uint32_t i, float coeff) { q_pbd(C, i, coeff); }
};

}  // namespace t10e

}  // namespace

}  // namespace xfem
