// Quadratic-hex element code of libxfem.so (sm_103a), shared by the H27
// mode (xfem_h27.cu) and meshes mixing T10s and H27s (xfem_qmixed.cu): GeoQuadratic3d on a hex mesh
// (XPBDFEM/Geo.cpp:836-1053). Every hex gets a node on each edge and face and
// one at its centre, numbered i + 3j + 9k on its 3x3x3 grid; SolveElement on
// ElementParamsQuadraticHex (XPBDFEM/Fem.cpp:871-897: SolveElementPixar
// :361-433 and SolveElementMixed :437-564 with Nodes = 27, PointsLo = 8 and
// PointsHi = 27; the cube models leave an H27 alone), SolveVolumeOnly on the
// 2x2x2 rule (:840-867), DampElement (:910-937) and PbdDamp
// (XPBDFEM/Xpbd.h:306-346), in the element kernel of xfem_elements.cuh.
//
// One warp per H27: an element's 27 nodes, its 703-value record and its 27
// quadrature points do not fit one thread. Lane n < 27 owns node n (its load,
// its share of the prefactored I1, its gradient rows, its update); lane p
// owns quadrature point p when the deformation gradients are formed. The
// node offsets P and each point's G Ji (the energy gradient mapped back to
// the reference frame) pass between the two through 3 KB of shared memory
// per warp, next to the warp's copy of the element's record. Sums over lanes
// are xor butterflies, so every lane holds the same bits and every lane takes
// the same branch.
//
// A pass is one warp's chain of some 1,300 instructions with 24 warps per SM.
// What shortened it (28,800 H27s, 20 substeps, 2,931 -> 1,763 us): the
// gradient tables in shared memory in the order each phase reads them, node
// offsets as one 16-byte read, three lanes per point on the 8-point rule, the
// prefactored row without branches, eight sums in one butterfly, and the next
// element's record and ids fetched while the pass ends.
//
// Records: 704 floats per H27 (the 703 of the reference's flattening, one
// pad), element-major, read by every lane of the element's warp. The
// gradient tables (the 2x2x2 rule's 648 floats, then the 3x3x3 rule's 2187)
// sit in el_tab.
#pragma once

#include "xfem_elements.cuh"

namespace xfem {

namespace {

namespace h27e {

constexpr int kJL = 0, kWL = 72, kJH = 80, kWH = 323, kQQ = 350, kQR = 376, kVol = 701, kArea = 702, kRec = 704;
constexpr int kTab8 = 0, kTab27 = 8 * 27 * 3;
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
	return v;
}

// N sums at once: their butterflies' latencies overlap.
template <int N>
__device__ __forceinline__ void wsums(float (&v)[N]) {
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
#pragma unroll
		for (int k = 0; k < N; k++) v[k] += __shfl_xor_sync(kAll, v[k], o);
}

// The gradient tables in shared memory, once per block: by node and point (a
// lane per point reads a node's row), and by point, axis and node (a lane per
// node reads a point's rows).
struct Tables {
	float4 a8[26][8], a27[26][27];
	float b8[8][3][32], b27[27][3][32];
};

__device__ __forceinline__ float tab(const DevCtx& C, int hi, int p, int n, int k) {
	return __ldg(C.el_tab + (hi ? kTab27 : kTab8) + (p * 27 + n) * 3 + k);
}

__device__ __forceinline__ void load_tables(const DevCtx& C, Tables& T) {
	for (uint32_t i = threadIdx.x; i < 27u * 32u; i += blockDim.x) {
		const int p = (int)(i / 32u), n = (int)(i % 32u);
		const float x = n < 27 ? tab(C, 1, p, n, 0) : 0.0f, y = n < 27 ? tab(C, 1, p, n, 1) : 0.0f,
		            z = n < 27 ? tab(C, 1, p, n, 2) : 0.0f;
		T.b27[p][0][n] = x, T.b27[p][1][n] = y, T.b27[p][2][n] = z;
		if (n < 26) T.a27[n][p] = make_float4(x, y, z, 0.0f);
		if (p < 8) {
			const float u = n < 27 ? tab(C, 0, p, n, 0) : 0.0f, v = n < 27 ? tab(C, 0, p, n, 1) : 0.0f,
			            w = n < 27 ? tab(C, 0, p, n, 2) : 0.0f;
			T.b8[p][0][n] = u, T.b8[p][1][n] = v, T.b8[p][2][n] = w;
			if (n < 26) T.a8[n][p] = make_float4(u, v, w, 0.0f);
		}
	}
	__syncthreads();
}

// per-warp scratch: the element's record (copied in once per element, so
// the lanes' scattered reads of it wait on shared memory, not on L2) and
// vertex ids, node offsets from node 26, and each point's G Ji, a row of three
// per axis, for the first and the second constraint
struct Scratch {
	float4 rec[kRec / 4];
	uint32_t vid[28];
	uint32_t have;  // the element whose record and ids are here or on their way
	uint32_t pad[3];
	float4 P[26];
	float4 M0[27][3], M1[27][3];
};

struct Elem {
	const float* R;  // the record (this warp's shared copy)
	const Tables* T;
	uint32_t lane;
	float4 O, D;  // this lane's node (lanes >= 27: zero)
	float w;
	uint32_t dv;
};

__device__ __forceinline__ float rec(const Elem& E, int j) { return E.R[j]; }

// P_n = (O_n - O_26) + (D_n - D_26) (solve), or O_n - O_26 (vmode)
__device__ __forceinline__ void share_rel(Scratch& s, const Elem& E, bool vmode) {
	const float ox = __shfl_sync(kAll, E.O.x, 26), oy = __shfl_sync(kAll, E.O.y, 26), oz = __shfl_sync(kAll, E.O.z, 26);
	const float dx = __shfl_sync(kAll, E.D.x, 26), dy = __shfl_sync(kAll, E.D.y, 26), dz = __shfl_sync(kAll, E.D.z, 26);
	__syncwarp();
	if (E.lane < 26)
		s.P[E.lane] = vmode ? make_float4(E.O.x - ox, E.O.y - oy, E.O.z - oz, 0.0f)
		                    : make_float4((E.O.x - ox) + (E.D.x - dx), (E.O.y - oy) + (E.D.y - dy),
		                                  (E.O.z - oz) + (E.D.z - dz), 0.0f);
	__syncwarp();
}

__device__ __forceinline__ float trace_xtx(const float F[3][3]) {
	return fmaf(F[0][0], F[0][0], fmaf(F[0][1], F[0][1], F[0][2] * F[0][2])) +
	       fmaf(F[1][0], F[1][0], fmaf(F[1][1], F[1][1], F[1][2] * F[1][2])) +
	       fmaf(F[2][0], F[2][0], fmaf(F[2][1], F[2][1], F[2][2] * F[2][2]));
}

// What a point computes (the per-point terms of SolveElementPixar and
// SolveElementMixed, XPBDFEM/Fem.cpp:379-427, 459-489, 532-549).
enum PointTerm {
	kHydro = 0,      // (J - a)^2 into slot 1
	kPixarFull = 1,  // I1 + hw (J - a)^2 (mu / 2 = 1) into slot 0
	kDev = 2,        // the deviatoric I1 (Mixed) or its Yeoh polynomial into slot 0
	kDevHydro = 3,   // kDev, and (J - a)^2 into slot 1
};

// The point terms over a rule (hi: the 27 points, else the 8) into M0 / M1;
// returns this lane's U contributions (summed by the caller). wscale scales
// every point's weight (a ring element's share of its ring volume); skin: the
// Yeoh constants of ContinuousSkin (XPBDFEM/Fem.cpp:994) instead of the
// body's.
template <int TERM>
__device__ __forceinline__ void points(const DevCtx& C, Scratch& s, const Elem& E, int hi, const BodyParams& bp,
                                       uint32_t e, float a, float& u0, float& u1, float wscale = 1.0f,
                                       bool skin = false) {
	u0 = u1 = 0.0f;
	// On the 27 points a lane takes one; on the 8 points three lanes share one,
	// lane p + 8 c forming column c of its F and row c of its G Ji.
	const int p = hi ? (int)E.lane : (int)(E.lane & 7u), own = hi ? 0 : (int)(E.lane >> 3);
	float Ji[3][3], F[3][3], A[3][3], G0[3][3], G1[3][3];
	const bool on = E.lane < (hi ? 27u : 24u);
	{
		const int pj = on ? p : 0, jb = (hi ? kJH : kJL) + 9 * pj;
#pragma unroll
		for (int c = 0; c < 3; c++)
#pragma unroll
			for (int r = 0; r < 3; r++) Ji[c][r] = rec(E, jb + 3 * c + r);
		if (hi) {
			float Dm[3][3] = {{0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}};
#pragma unroll 2
			for (int n = 0; n < 26; n++) {
				const float4 x = s.P[n], d = E.T->a27[n][pj];
				Dm[0][0] = fmaf(d.x, x.x, Dm[0][0]), Dm[1][0] = fmaf(d.x, x.y, Dm[1][0]), Dm[2][0] = fmaf(d.x, x.z, Dm[2][0]);
				Dm[0][1] = fmaf(d.y, x.x, Dm[0][1]), Dm[1][1] = fmaf(d.y, x.y, Dm[1][1]), Dm[2][1] = fmaf(d.y, x.z, Dm[2][1]);
				Dm[0][2] = fmaf(d.z, x.x, Dm[0][2]), Dm[1][2] = fmaf(d.z, x.y, Dm[1][2]), Dm[2][2] = fmaf(d.z, x.z, Dm[2][2]);
			}
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) F[c][r] = fmaf(Ji[0][r], Dm[c][0], fmaf(Ji[1][r], Dm[c][1], Ji[2][r] * Dm[c][2]));
		} else {
			const float* Pc = reinterpret_cast<const float*>(s.P) + (own < 3 ? own : 0);
			float Dm[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
			for (int n = 0; n < 26; n++) {
				const float x = Pc[4 * n];
				const float4 d = E.T->a8[n][p];
				Dm[0] = fmaf(d.x, x, Dm[0]);
				Dm[1] = fmaf(d.y, x, Dm[1]);
				Dm[2] = fmaf(d.z, x, Dm[2]);
			}
			float Fc[3];
#pragma unroll
			for (int r = 0; r < 3; r++) Fc[r] = fmaf(Ji[0][r], Dm[0], fmaf(Ji[1][r], Dm[1], Ji[2][r] * Dm[2]));
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) F[c][r] = __shfl_sync(kAll, Fc[r], p + 8 * c);
		}
	}
	if (on) {
		const float wt = wscale * rec(E, (hi ? kWH : kWL) + p);
		const float J = adj_det(F, A);
		const float Ja = J - a;
		if (TERM == kHydro || TERM == kDevHydro) {
			u1 = wt * Ja * Ja;
			const float s1 = 2.0f * wt * Ja;
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) G1[c][r] = A[c][r] * s1;
		}
		if (TERM == kPixarFull) {
			const float hw = __ldg(&bp.hw);
			u0 = wt * fmaf(hw * Ja, Ja, trace_xtx(F));
			const float s1 = 2.0f * wt, s2 = 2.0f * wt * hw * Ja;
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) G0[c][r] = fmaf(F[r][c], s1, A[c][r] * s2);
		}
		if (TERM == kDev || TERM == kDevHydro) {
			const float I1 = trace_xtx(F);
			float sc;
			if (e == 3u) {
				u0 = wt * I1;
				sc = 2.0f * wt;
			} else {
				const float C0 = skin ? 0.1095f : __ldg(&bp.yeoh[0]), C1 = skin ? 14.95f : __ldg(&bp.yeoh[1]),
				            C2 = skin ? 4.595f : __ldg(&bp.yeoh[2]);
				const float IM = I1 - 3.0f;
				u0 = wt * (IM * fmaf(IM, fmaf(IM, C2, C1), C0));
				sc = 2.0f * wt * fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
			}
#pragma unroll
			for (int c = 0; c < 3; c++)
#pragma unroll
				for (int r = 0; r < 3; r++) G0[c][r] = F[r][c] * sc;
		}
		// M[j][r] = sum_k G[k][r] Ji[j][k]
		auto row = [&](const float G[3][3], const float J[3]) {
			return make_float4(fmaf(G[0][0], J[0], fmaf(G[1][0], J[1], G[2][0] * J[2])),
			                   fmaf(G[0][1], J[0], fmaf(G[1][1], J[1], G[2][1] * J[2])),
			                   fmaf(G[0][2], J[0], fmaf(G[1][2], J[1], G[2][2] * J[2])), 0.0f);
		};
		if (hi) {
#pragma unroll
			for (int j = 0; j < 3; j++) {
				if (TERM != kHydro) s.M0[p][j] = row(G0, Ji[j]);
				if (TERM == kHydro || TERM == kDevHydro) s.M1[p][j] = row(G1, Ji[j]);
			}
		} else {
			const float Jc[3] = {own == 0 ? Ji[0][0] : own == 1 ? Ji[1][0] : Ji[2][0],
			                     own == 0 ? Ji[0][1] : own == 1 ? Ji[1][1] : Ji[2][1],
			                     own == 0 ? Ji[0][2] : own == 1 ? Ji[1][2] : Ji[2][2]};
			if (TERM != kHydro) s.M0[p][own] = row(G0, Jc);
			if (TERM == kHydro || TERM == kDevHydro) s.M1[p][own] = row(G1, Jc);
			if (own) u0 = u1 = 0.0f;  // one lane's share per point
		}
	}
	__syncwarp();
}

// g_n += sum_p M_p dN_p[n] for this lane's node (n < 26) from slot M
__device__ __forceinline__ Vec3 gather(const float4 (*M)[3], const Elem& E, int hi) {
	Vec3 g = {0.0f, 0.0f, 0.0f};
	const float(*T)[3][32] = hi ? E.T->b27 : E.T->b8;
	const int np = hi ? 27 : 8, n = (int)E.lane;
	if (n < 26)
#pragma unroll 4
		for (int p = 0; p < np; p++) {
			const float d0 = T[p][0][n], d1 = T[p][1][n], d2 = T[p][2][n];
			const float4 a = M[p][0], b = M[p][1], c = M[p][2];
			g.x += fmaf(a.x, d0, fmaf(b.x, d1, c.x * d2));
			g.y += fmaf(a.y, d0, fmaf(b.y, d1, c.y * d2));
			g.z += fmaf(a.z, d0, fmaf(b.z, d1, c.z * d2));
		}
	return g;
}

// node 26 takes minus the others' sum s
__device__ __forceinline__ Vec3 root_of(const Elem& E, const Vec3& g, const float* s) {
	return E.lane == 26 ? Vec3{g.x - s[0], g.y - s[1], g.z - s[2]} : E.lane < 26 ? g : Vec3{0.0f, 0.0f, 0.0f};
}

// The gradient with node 26's from the others' sum; u (this lane's energy
// contribution) summed over the lanes.
__device__ __forceinline__ Vec3 root_u(const Elem& E, const Vec3& g, float& u) {
	const bool on = E.lane < 26;
	float v[4] = {on ? g.x : 0.0f, on ? g.y : 0.0f, on ? g.z : 0.0f, u};
	wsums(v);
	u = v[3];
	return root_of(E, g, v);
}

// The same for two gradients and energies together.
__device__ __forceinline__ void root2_u(const Elem& E, Vec3& g0, float& u0, Vec3& g1, float& u1) {
	const bool on = E.lane < 26;
	float v[8] = {on ? g0.x : 0.0f, on ? g0.y : 0.0f, on ? g0.z : 0.0f, u0,
	              on ? g1.x : 0.0f, on ? g1.y : 0.0f, on ? g1.z : 0.0f, u1};
	wsums(v);
	u0 = v[3];
	u1 = v[7];
	g0 = root_of(E, g0, v);
	g1 = root_of(E, g1, v + 4);
}

// The prefactored I1 over the 26 offsets (XPBDFEM/Fem.cpp:163-192): this
// lane's gradient row (without node 26's) and its share of U.
__device__ __forceinline__ float pref_row(const Scratch& s, const Elem& E, Vec3& g) {
	float u = 0.0f;
	g = {0.0f, 0.0f, 0.0f};
	const int i = (int)E.lane;
	if (i < 26) {
		const float qq = rec(E, kQQ + i);
		const Vec3 Pi = v3(s.P[i]);
		u = qq * dot(Pi, Pi);
		g = {2.0f * qq * Pi.x, 2.0f * qq * Pi.y, 2.0f * qq * Pi.z};
		// QR of the pair (lo, hi), lo < hi: row lo starts at lo (51 - lo) / 2.
		// No branches: the pair's place is selected, and j = i adds 0 P_i.
		const int below = kQR + i - 1;                       // + j (51 - j) / 2 - j: pairs (j, i)
		const int above = kQR + i * (51 - i) / 2 - i - 1;  // + j: pairs (i, j)
#pragma unroll
		for (int j = 0; j < 26; j++) {
			const Vec3 Pj = v3(s.P[j]);
			const float q = E.R[j < i ? below + (j * (51 - j) / 2 - j) : above + j];
			const float qr = j == i ? 0.0f : q;
			g = {fmaf(qr, Pj.x, g.x), fmaf(qr, Pj.y, g.y), fmaf(qr, Pj.z, g.z)};
			const float un = fmaf(qr, dot(Pi, Pj), u);
			u = j > i ? un : u;
		}
	}
	return u;
}

__device__ __forceinline__ float wgg_of(const Elem& E, const Vec3& a, const Vec3& b) {
	return 1.0e-22f + wsum(E.lane < 27 ? E.w * dot(a, b) : 0.0f);
}
__device__ __forceinline__ void wgg3_of(const Elem& E, const Vec3& g0, const Vec3& g1, float& s00, float& s10, float& s11) {
	const bool on = E.lane < 27;
	float v[3] = {on ? E.w * dot(g0, g0) : 0.0f, on ? E.w * dot(g1, g0) : 0.0f, on ? E.w * dot(g1, g1) : 0.0f};
	wsums(v);
	s00 = 1.0e-22f + v[0];
	s10 = 1.0e-22f + v[1];
	s11 = 1.0e-22f + v[2];
}
__device__ __forceinline__ float gD_of(const Elem& E, const Vec3& g) {
	return wsum(E.lane < 27 ? fmaf(g.x, E.D.x, fmaf(g.y, E.D.y, g.z * E.D.z)) : 0.0f);
}
__device__ __forceinline__ void move(Elem& E, float l, const Vec3& g) {
	const float s = E.w * l;
	E.D.x = fmaf(s, g.x, E.D.x);
	E.D.y = fmaf(s, g.y, E.D.y);
	E.D.z = fmaf(s, g.z, E.D.z);
}
__device__ __forceinline__ void move2(Elem& E, float l0, const Vec3& g0, float l1, const Vec3& g1) {
	const float s0 = E.w * l0, s1 = E.w * l1;
	E.D.x = fmaf(s1, g1.x, fmaf(s0, g0.x, E.D.x));
	E.D.y = fmaf(s1, g1.y, fmaf(s0, g0.y, E.D.y));
	E.D.z = fmaf(s1, g1.z, fmaf(s0, g0.z, E.D.z));
}

// Where a block's dynamic shared memory holds this mode's part (after the
// T10s' on meshes mixing both).
#ifndef XFEM_H27_SMEM_AT
#define XFEM_H27_SMEM_AT 0
#endif
struct Shared {
	Tables t;
	Scratch s[8];  // 256-thread blocks: 8 warps
};
__device__ __forceinline__ Shared& shared() {
	extern __shared__ __align__(128) unsigned char h27_smem[];
	return *reinterpret_cast<Shared*>(h27_smem + XFEM_H27_SMEM_AT);
}

// Starts the copy of element i's record and vertex ids into the warp's
// scratch (asynchronous 16-byte copies: a warp's next element is known, so
// its 2.9 KB come while the pass ends and the barrier is waited for).
__device__ __forceinline__ void fetch(const DevCtx& C, uint32_t i, Scratch& s, uint32_t lane) {
	__syncwarp();  // every lane is done with the last element's copy
	const float4* src = C.el_rec + (size_t)i * (kRec / 4);
	auto copy = [](void* dst, const void* from) {
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(from) : "memory");
	};
	for (uint32_t k = lane; k < kRec / 4; k += 32) copy(&s.rec[k], src + k);
	if (lane < 7u) copy(&s.vid[4 * lane], C.el_vid + 7 * (size_t)i + lane);
	if (lane == 0) s.have = i;
	__syncwarp();
}

__device__ __forceinline__ void load(const DevCtx& C, uint32_t i, Scratch& s, const Tables& T, Elem& E) {
	E.lane = threadIdx.x & 31u;
	E.T = &T;
	if (s.have != i) {
		asm volatile("cp.async.wait_all;" ::: "memory");  // a fetch that is not used after all
		fetch(C, i, s, E.lane);
	}
	asm volatile("cp.async.wait_all;" ::: "memory");
	__syncwarp();
	E.R = reinterpret_cast<const float*>(s.rec);
	E.O = E.D = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
	E.w = 0.0f;
	E.dv = 0;
	if (E.lane < 27) {
		E.dv = s.vid[E.lane];
		ld_vertex(C.vert + 2 * (size_t)E.dv, E.O, E.D);
		E.w = E.O.w;
	}
}

// One H27 of a pass (the kinds of ElemPass), every lane of the warp; next: the
// element to fetch for the warp's next call (kNoElem: none).
template <int KIND>
__device__ __noinline__ void h27_pass(const DevCtx& C, uint32_t i, uint32_t next, float inv_dt, float inv_dt2, float rd) {
	Scratch& s = shared().s[threadIdx.x >> 5];
	Elem E;
	load(C, i, s, shared().t, E);
	const BodyParams& bp = C.bodies[__float_as_uint(__shfl_sync(kAll, E.D.w, 0)) >> 8];
	const uint32_t e = __ldg(&bp.energy);
	if (KIND != kVolume && (e == 11u || e == 12u)) return;  // SolveElementCube acts on 8-node hexes only
	const float vol = rec(E, kVol);
	const uint32_t type = __ldg(&bp.rayleigh_type);
	const float damp = KIND == kSolve && type < 2u ? __ldg(&bp.damping) : 0.0f;
	const bool limit = type == 1u;
	const bool sim = __ldg(&bp.simultaneous) != 0u;
	share_rel(s, E, KIND == kRayleigh);
	float u0, u1;
	if (KIND == kVolume) {
		points<kHydro>(C, s, E, 0, bp, e, 1.0f, u0, u1);
		const Vec3 g = root_u(E, gather(s.M1, E, 0), u1);
		const float U = u1;
		const float alpha = __ldg(&bp.compliance) * vol * inv_dt2;
		move(E, (-2.0f * U) / fmaf(2.0f * U, alpha, wgg_of(E, g, g)), g);
	} else if (e <= 2u) {
		float U;
		Vec3 g;
		if (e != 2u) {
			const int hi = e == 0u;
			points<kPixarFull>(C, s, E, hi, bp, e, __ldg(&bp.a), u0, u1);
			g = root_u(E, gather(s.M0, E, hi), u0);
			U = u0;
		} else {
			const float hw = __ldg(&bp.hw);
			points<kHydro>(C, s, E, 0, bp, e, __ldg(&bp.a), u0, u1);
			Vec3 gh = gather(s.M1, E, 0), gi;
			float UI = pref_row(s, E, gi);
			root2_u(E, gh, u1, gi, UI);
			U = fmaf(hw, u1, UI);
			g = {fmaf(hw, gh.x, gi.x), fmaf(hw, gh.y, gi.y), fmaf(hw, gh.z, gi.z)};
		}
		const float comp = __ldg(&bp.compliance) / vol;
		const float wgg = wgg_of(E, g, g);
		if (KIND == kRayleigh)
			move(E, -gD_of(E, g) / fmaf(2.0f * U, comp * inv_dt / rd, wgg), g);
		else
			move(E, lambda1_of(U, wgg, damp > 0.0f ? gD_of(E, g) : 0.0f, comp * inv_dt2, comp, damp, limit, inv_dt), g);
	} else {
		const float a = __ldg(&bp.a);
		const float comp0 = __ldg(&bp.inv_mu) / vol, comp1 = __ldg(&bp.inv_lambda) / vol;
		const float alpha0 = comp0 * inv_dt2, alpha1 = comp1 * inv_dt2;
		const bool coupled = KIND == kRayleigh || sim;
		const bool full = full_quadrature(e);
		float U0, U1 = 0.0f;
		Vec3 g0, g1 = {0.0f, 0.0f, 0.0f};
		if (full) {
			if (coupled && e != 6u) {
				points<kDevHydro>(C, s, E, 1, bp, e, a, u0, U1);
				g0 = gather(s.M0, E, 1);
				g1 = gather(s.M1, E, 1);
				root2_u(E, g0, u0, g1, U1);
			} else {
				points<kDev>(C, s, E, 1, bp, e, a, u0, u1);
				g0 = root_u(E, gather(s.M0, E, 1), u0);
			}
			U0 = fmaxf(0.0001f, u0);
		} else {
			U0 = pref_row(s, E, g0);
			if (coupled) {
				points<kHydro>(C, s, E, 0, bp, e, a, u0, U1);
				g1 = gather(s.M1, E, 0);
				root2_u(E, g0, U0, g1, U1);
			} else {
				g0 = root_u(E, g0, U0);
			}
			if (e == 7u) {
				const float C0 = __ldg(&bp.yeoh[0]), C1 = __ldg(&bp.yeoh[1]), C2 = __ldg(&bp.yeoh[2]);
				const float IM = U0 - 3.0f;
				U0 = fmaxf(0.0001f, IM * fmaf(IM, fmaf(IM, C2, C1), C0));
				const float gs = fmaf(IM, fmaf(IM, 3.0f * C2, 2.0f * C1), C0);
				g0 = {g0.x * gs, g0.y * gs, g0.z * gs};
			}
		}
		if (coupled) {
			if (e == 6u) {
				__syncwarp();
				points<kHydro>(C, s, E, 0, bp, e, a, u0, U1);
				g1 = root_u(E, gather(s.M1, E, 0), U1);
			}
			float wgg0, wgg1, wgg2;
			wgg3_of(E, g0, g1, wgg0, wgg1, wgg2);
			float l0, l1;
			if (KIND == kRayleigh) {
				if (sim) {
					cramer(fmaf(2.0f * U0, comp0 * inv_dt / rd, wgg0), wgg1, fmaf(2.0f * U1, comp1 * inv_dt / rd, wgg2),
					       -gD_of(E, g0), -gD_of(E, g1), l0, l1);
					move2(E, l0, g0, l1, g1);
				} else {
					move(E, -gD_of(E, g0) / fmaf(2.0f * U0, comp0 * inv_dt / rd, wgg0), g0);
					move(E, -gD_of(E, g1) / fmaf(2.0f * U1, comp1 * inv_dt / rd, wgg2), g1);
				}
			} else {
				const bool dm = damp > 0.0f;
				lambda2_of(U0, U1, wgg0, wgg1, wgg2, dm ? gD_of(E, g0) : 0.0f, dm ? gD_of(E, g1) : 0.0f, alpha0, alpha1,
				           comp0, comp1, damp, limit, inv_dt, l0, l1);
				move2(E, l0, g0, l1, g1);
			}
		} else {
			// serial: deviatoric, refresh P, hydrostatic (XPBDFEM/Fem.cpp:490-521, 532-551)
			const float wgg0 = wgg_of(E, g0, g0);
			move(E, lambda1_of(U0, wgg0, damp > 0.0f ? gD_of(E, g0) : 0.0f, alpha0, comp0, damp, limit, inv_dt), g0);
			share_rel(s, E, false);
			const int hi = full && e != 6u;
			points<kHydro>(C, s, E, hi, bp, e, a, u0, U1);
			g1 = root_u(E, gather(s.M1, E, hi), U1);
			const float wgg2 = wgg_of(E, g1, g1);
			move(E, lambda1_of(U1, wgg2, damp > 0.0f ? gD_of(E, g1) : 0.0f, alpha1, comp1, damp, limit, inv_dt), g1);
		}
	}
	if (next != kNoElem) fetch(C, next, s, E.lane);
	if (E.lane < 27) st_vertex(C.vert + 2 * (size_t)E.dv, E.O, E.D);
}

// PbdDamp over the 27 nodes (XPBDFEM/Xpbd.h:306-346) on the canonical state
// (O = X, D = V), the coefficient coeff / surfaceArea capped at 1.
__device__ __forceinline__ void h27_pbd_in(const DevCtx& C, Scratch& s, const Tables& T, uint32_t i, float coeff) {
	Elem E;
	load(C, i, s, T, E);
	const bool node = E.lane < 27;
	const float damping = fminf(1.0f, coeff / rec(E, kArea));
	const float Wavg = (1.0e-8f + wsum(E.w)) * (1.0f / 27.0f), Wmin = 0.0001f * Wavg;
	const float rx = __shfl_sync(kAll, E.O.x, 26), ry = __shfl_sync(kAll, E.O.y, 26), rz = __shfl_sync(kAll, E.O.z, 26);
	const Vec3 x = {E.O.x - rx, E.O.y - ry, E.O.z - rz};
	const float M = node ? Wavg / fmaxf(Wmin, E.w) : 0.0f;
	const float im = 1.0f / wsum(M);
	const Vec3 xcm = {wsum(x.x * M) * im, wsum(x.y * M) * im, wsum(x.z * M) * im};
	const Vec3 vcm = {wsum(E.D.x * M) * im, wsum(E.D.y * M) * im, wsum(E.D.z * M) * im};
	const Vec3 r = {x.x - xcm.x, x.y - xcm.y, x.z - xcm.z};
	const Vec3 c = cross(r, v3(E.D));
	const Vec3 L = {wsum(M * c.x), wsum(M * c.y), wsum(M * c.z)};
	const float xx = r.x * r.x, yy = r.y * r.y, zz = r.z * r.z;
	const float I00 = wsum(M * (yy + zz)), I11 = wsum(M * (xx + zz)), I22 = wsum(M * (xx + yy));
	const float I01 = -wsum(M * (r.x * r.y)), I12 = -wsum(M * (r.y * r.z)), I02 = -wsum(M * (r.z * r.x));
	const float a00 = fmaf(I11, I22, -I12 * I12), a01 = fmaf(I02, I12, -I01 * I22), a02 = fmaf(I01, I12, -I02 * I11);
	const float a11 = fmaf(I00, I22, -I02 * I02), a12 = fmaf(I01, I02, -I00 * I12), a22 = fmaf(I00, I11, -I01 * I01);
	const float idet = 1.0f / fmaf(I00, a00, fmaf(I01, a01, I02 * a02));
	const Vec3 om = {fmaf(a00, L.x, fmaf(a01, L.y, a02 * L.z)) * idet, fmaf(a01, L.x, fmaf(a11, L.y, a12 * L.z)) * idet,
	                 fmaf(a02, L.x, fmaf(a12, L.y, a22 * L.z)) * idet};
	const Vec3 cr = cross(om, r);
	E.D.x = fmaf(damping, (vcm.x + cr.x) - E.D.x, E.D.x);
	E.D.y = fmaf(damping, (vcm.y + cr.y) - E.D.y, E.D.y);
	E.D.z = fmaf(damping, (vcm.z + cr.z) - E.D.z, E.D.z);
	if (node) st_vertex(C.vert + 2 * (size_t)E.dv, E.O, E.D);
}

__device__ __noinline__ void h27_pbd(const DevCtx& C, uint32_t i, float coeff) {
	h27_pbd_in(C, shared().s[threadIdx.x >> 5], shared().t, i, coeff);
}

struct H27Elem {
	static constexpr int kLanes = 32, kPbdLanes = 32;
	static constexpr int kBlock = 256;
	static constexpr int kMinBlocks = 3;  // at most 85 registers: three 256-thread blocks per SM
	static constexpr uint32_t kVid4 = 7;
	static constexpr size_t smem() { return sizeof(Shared); }
	__device__ static void init(const DevCtx& C) {
		if ((threadIdx.x & 31u) == 0u) shared().s[threadIdx.x >> 5].have = kNoElem;
		load_tables(C, shared().t);
	}
	template <int KIND>
	__device__ static void pass(const DevCtx& C, uint32_t i, uint32_t, bool, float inv_dt, float inv_dt2, float rd,
	                            uint32_t next = kNoElem, uint32_t = 0) {
		h27_pass<KIND>(C, i, next, inv_dt, inv_dt2, rd);
	}
	__device__ static void pbd(const DevCtx& C, uint32_t i, float coeff) { h27_pbd(C, i, coeff); }
};

}  // namespace h27e

}  // namespace

}  // namespace xfem
