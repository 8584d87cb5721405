// One resident chunk of a colour pass: the solve, volume and damping sweeps of
// a warp's 32 clusters, shared by the launch forms of xfem_kernels.cu and the
// one-cluster form of xfem_cluster.cu. Internal linkage: each translation unit
// gets its own copy.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "xfem_device.cuh"
#include "xfem_internal.h"

namespace xfem {

namespace {

__device__ __forceinline__ int tip_at(const DevCtx& C, uint32_t v, bool first) {
	return first ? -1 : __ldg(C.tip_of + v);
}

// Adjoint tape: the owner of a vertex records O right after the advance
// (the position the substep starts from, with the inverse mass the solves
// use) and D right before it, in one 32-byte sector, and, from the second
// substep of a launch on, the tip trajectory (O is then the position after
// the previous substep). q: the vertex's tip or -1 (tip_at), read ahead: read
// here, each of a lane's vertices waited for it in turn (12,288 tets, 200
// substeps: 6.80 ms, 6.10 so).
__device__ __forceinline__ void tape_vertex(const DevCtx& C, uint32_t v, const float4& O, const float4& Dbefore,
                                            uint32_t s, int q) {
	float4* p = C.tape_v + 2 * ((size_t)s * C.nverts + v);
	__stcs(p, O);
	__stcs(p + 1, Dbefore);
	if (q >= 0) C.traj[(size_t)(C.sub_base + s - 1) * C.ntips + q] = O;
}

// Adjoint tape: the input displacement of one solve's four vertices.
__device__ __forceinline__ void tape_tet(const DevCtx& C, uint32_t s, uint32_t row, uint32_t lane, const float4 D[4]) {
	float4* p = C.tape_t + ((size_t)s * C.ntrows + row) * 3 * kLanes + lane;
	__stcs(p, make_float4(D[0].x, D[0].y, D[0].z, D[1].x));
	__stcs(p + kLanes, make_float4(D[1].y, D[1].z, D[2].x, D[2].y));
	__stcs(p + 2 * kLanes, make_float4(D[2].z, D[3].x, D[3].y, D[3].z));
}

// ---- damping after the velocity update (GeoLinear3d::Damp) ------------------
// State during the damping sweeps: vert[2v] = (X, w), vert[2v+1] = (V, bits).

// How a body's tets are damped at this tick (XPBDFEM/Geo.cpp:346-352, 792-798):
// with which Rayleigh ratio or PBD coefficient, and which of them: the
// amortized type damps one eighth of the body's order per tick, x 8.
struct DampBody {
	bool on, amort;
	float rayleigh, pbd;
	uint32_t lo, hi;  // amortized: the slice of the body's order
};

__device__ __forceinline__ DampBody damp_of(const BodyParams& bp, uint32_t tick, int kind) {
	DampBody d = {false, __ldg(&bp.rayleigh_type) == 3u, 0.0f, 0.0f, 0u, 0u};
	if (kind == 0) {
		d.rayleigh = __ldg(&bp.damping) * (d.amort ? 8.0f : 1.0f);
		d.on = __ldg(&bp.rayleigh_type) >= 2u && d.rayleigh > 0.0f;
	} else {
		d.on = __ldg(&bp.pbd_on) != 0u;
		d.pbd = d.amort ? __ldg(&bp.pbd_coeff_amortized) : __ldg(&bp.pbd_coeff);
	}
	const uint32_t nt = __ldg(&bp.ntets), m = tick % 8u;
	d.lo = nt * m / 8u;
	d.hi = nt * (m + 1u) / 8u;
	return d;
}

// Whether the plain kernels' solve is this body's: a coupled or serial
// MixedSel or Yeoh without in-solve damping.
__device__ __forceinline__ bool plain_solve(const Mat& m) {
	return (m.model == kModelNeo || m.model == kModelYeoh) && !(m.damp > 0.0f);
}

// Header word of a cluster lane: nv | nt << 4 | advance mask << 8 | body << 16.
// A vertex is advanced (previous substep finalized, next one predicted) by
// the lowest-colour cluster touching it, just before that cluster's solve.

template <bool LAMBDAS, bool TAPE, bool EXT, bool XSOLVE, class VS, class BP>
__device__ __forceinline__ void run_chunk_cube(const DevCtx& C, const VS& vs, const BP& bps, Stage& st, int next, const uint4& mnext, uint32_t lane,
                                               bool first, float dt, float inv_dt, float inv_dt2, uint32_t trow,
                                               uint32_t s_launch, uint32_t chunk, bool finish_last) {
	const float4* rec = reinterpret_cast<const float4*>(st.buf);
	const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(st.buf + 2048u * 6u);
	const uint32_t* vids = hdrs + kLanes;
	const uint32_t hdr = hdrs[lane];
	const bool live = (hdr & 15u) != 0;
	const uint32_t mask = (hdr >> 8) & 0xffu;
	uint32_t vid[8];
	float4 O[8], D[8];
	// With damping sweeps, the vertices whose last solve of the substep this
	// is: it finishes them (to the canonical X, V that the sweeps work on).
	// Loaded ahead of the solves: after them it was an L2 trip on the chain.
	uint32_t last = 0u;
	if (live) {
		const Mat mat = bps.mat(C, hdr >> 16);
		if (EXT && finish_last && mat.nvol == 0u)  // (else the body's last volume pass does)
			last = __ldg(C.lastmask + (size_t)chunk * kLanes + lane);
#pragma unroll
		for (int s = 0; s < 8; s++) vid[s] = vids[s * kLanes + lane];
		int tip[8];
		if (TAPE)
#pragma unroll
			for (int s = 0; s < 8; s++) tip[s] = (mask & (1u << s)) ? tip_at(C, vid[s], first) : -1;
#pragma unroll
		for (int s = 0; s < 8; s++) vs.ld(C, vid[s], O[s], D[s]);
#pragma unroll
		for (int s = 0; s < 8; s++)
			if (mask & (1u << s)) {
				const float4 Dbefore = D[s];
				bps.advance(C, vid[s], O[s], D[s], first, dt, inv_dt);
				if (TAPE) tape_vertex(C, vid[s], O[s], Dbefore, s_launch, tip[s]);
			}
		auto before = [&](int t, const float4* Dt) {
			if (TAPE) tape_tet(C, s_launch, trow + t, lane, Dt);
		};
		auto after = [&](int t, const float2& lam) {
			if (LAMBDAS) C.tlam[(size_t)(trow + t) * kLanes + lane] = lam;
		};
		// the extended kernel's solve only where the body needs it: its code
		// made the pass of a warp 40% longer (7,090 cycles against 5,060)
		if (XSOLVE && mat.model == kModelNone) {
			// the cube models leave a tet alone: the loop over the six would only
			// move the vertices around (36,864 cubes, 20 substeps: 714 -> 656 us)
			for (int t = 0; t < 6; t++) after(t, make_float2(0.0f, 0.0f));
		} else if (XSOLVE && !plain_solve(mat))
			solve_cube<XSOLVE>(mat, rec + lane, inv_dt, inv_dt2, O, D, before, after);
		else
			solve_cube<false, VS::kAhead && !TAPE>(mat, rec + lane, inv_dt, inv_dt2, O, D, before, after);
	}
	if (next >= 0) stage_issue_m(C, st, (uint32_t)next, mnext, lane);  // buffer consumed: prefetch
	if (live) {
		// O changes only where this cluster advanced or finished the vertex
		// (then the whole 32-byte state is stored); no other cluster of the
		// pass touches these vertices
#pragma unroll
		for (int s = 0; s < 8; s++) {
			if (EXT && (last & (1u << s))) bps.finalize(C, vid[s], O[s], D[s], inv_dt);
			if ((mask | last) & (1u << s))
				vs.st(C, vid[s], O[s], D[s]);
			else  // only D moved: a 16-byte store
				vs.st_d(C, vid[s], D[s]);
		}
	}
}

// One warp processes one resident chunk; lane = cluster. `next` >= 0 is the
// warp's next chunk: its copy is issued as soon as this chunk's records have
// been consumed, so it overlaps the write-back and what follows. EXT: the
// sweeps of the extended kernels; XSOLVE: some body's solve is the extended
// one (not plain_solve); a kernel compiled without it runs the small damped
// bodies of the interactive settings in 578 us against 621 for ten frames.
template <bool LAMBDAS, bool TAPE = false, bool EXT = false, bool XSOLVE = EXT, class VS, class BP>
__device__ __forceinline__ void run_chunk(const DevCtx& C, const VS& vs, const BP& bps, Stage& st, uint32_t chunk, int next, uint32_t lane, bool first,
                                          float dt, float inv_dt, float inv_dt2, uint32_t s_launch = 0,
                                          bool finish_last = false) {
	// the staged chunk's descriptor came with its copy; the next one's is
	// loaded now, off the critical path of the prefetch
	const uint4 m = st.meta;
	const uint4 mnext = next >= 0 ? __ldg(reinterpret_cast<const uint4*>(C.chunks) + next) : make_uint4(0u, 0u, 0u, 0u);
	const uint32_t ntmax = m.z & 0xffu, nvmax = (m.z >> 8) & 0xffu, trow = m.w;
	if (m.z & kShapeCube) {
		run_chunk_cube<LAMBDAS, TAPE, EXT, XSOLVE>(C, vs, bps, st, next, mnext, lane, first, dt, inv_dt, inv_dt2, trow, s_launch, chunk,
		                                            finish_last);
		return;
	}
	const float4* rec = reinterpret_cast<const float4*>(st.buf);
	const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(st.buf + 2048u * ntmax);
	const uint32_t* vids = hdrs + kLanes;
	const uint32_t* slots = vids + kLanes * nvmax;
	const uint32_t hdr = hdrs[lane];
	const uint32_t nv = hdr & 15u, nt = (hdr >> 4) & 15u, mask = (hdr >> 8) & 0xffu;
	float4* sO = st.vs + lane;
	float4* sD = st.vs + kLanes * nvmax + lane;
	uint32_t vid[kMaxClusterVerts];
	bool fin = false;
	if (nv) {
		const Mat mat = bps.mat(C, hdr >> 16);
		fin = EXT && finish_last && mat.nvol == 0u;
#pragma unroll
		for (uint32_t s = 0; s < kMaxClusterVerts; s++)
			if (s < nv) vid[s] = vids[s * kLanes + lane];
#pragma unroll
		for (uint32_t s = 0; s < kMaxClusterVerts; s++) {
			if (s < nv) {
				const int tip = TAPE && (mask & (1u << s)) ? tip_at(C, vid[s], first) : -1;
				float4 O, D;
				vs.ld(C, vid[s], O, D);
				if (mask & (1u << s)) {
					const float4 Dbefore = D;
					bps.advance(C, vid[s], O, D, first, dt, inv_dt);
					if (TAPE) tape_vertex(C, vid[s], O, Dbefore, s_launch, tip);
				}
				sO[s * kLanes] = O;
				sD[s * kLanes] = D;
			}
		}
		for (uint32_t t = 0; t < nt; t++) {
			const float4* r = rec + t * 4 * kLanes + lane;
			const TetRec tr = {r[0], r[kLanes], r[2 * kLanes], r[3 * kLanes]};
			const uint32_t sl = slots[t * kLanes + lane];
			const uint32_t s0 = sl & 15u, s1 = (sl >> 4) & 15u, s2 = (sl >> 8) & 15u, s3 = (sl >> 12) & 15u;
			const float4 O[4] = {sO[s0 * kLanes], sO[s1 * kLanes], sO[s2 * kLanes], sO[s3 * kLanes]};
			float4 D[4] = {sD[s0 * kLanes], sD[s1 * kLanes], sD[s2 * kLanes], sD[s3 * kLanes]};
			if (TAPE) tape_tet(C, s_launch, trow + t, lane, D);
			const float2 lam = XSOLVE && !plain_solve(mat) ? solve_tet<XSOLVE>(mat, tr, inv_dt, inv_dt2, O, D)
			                                            : solve_tet<false>(mat, tr, inv_dt, inv_dt2, O, D);
			sD[s0 * kLanes] = D[0];
			sD[s1 * kLanes] = D[1];
			sD[s2 * kLanes] = D[2];
			sD[s3 * kLanes] = D[3];
			if (LAMBDAS) C.tlam[(size_t)(trow + t) * kLanes + lane] = lam;
		}
	}
	if (next >= 0) stage_issue_m(C, st, (uint32_t)next, mnext, lane);  // buffer consumed: prefetch
	if (nv) {
		const uint32_t last = fin ? __ldg(C.lastmask + (size_t)chunk * kLanes + lane) : 0u;
#pragma unroll
		for (uint32_t s = 0; s < kMaxClusterVerts; s++) {
			if (s < nv) {
				float4 O = sO[s * kLanes], D = sD[s * kLanes];
				if (EXT && (last & (1u << s))) bps.finalize(C, vid[s], O, D, inv_dt);
				vs.st(C, vid[s], O, D);
			}
		}
	}
}

// Volume sweep k (1-based) over a resident chunk: SolveElementVolume on each
// tet of the cluster in order (GeoLinear3d::Constrain, XPBDFEM/Geo.cpp:
// 780-783), for lanes whose body runs at least k volume passes. The state is
// (O, D), as in the solve sweep; only D changes, except that with damping
// sweeps (finish) the body's last volume sweep finishes the vertices whose
// last solve this cluster makes. CUBE: canonical cube chunks, all in
// registers. Not inlined, like the damping passes.
template <bool CUBE, class VS>
__device__ __noinline__ void vol_chunk(const DevCtx& C, const VS& vs, Stage& st, uint32_t chunk, uint32_t ntmax, uint32_t nvmax,
                                       int next, uint32_t lane, float inv_dt, float inv_dt2, uint32_t k, bool finish) {
	constexpr uint32_t NV = CUBE ? 8u : kMaxClusterVerts;
	const float4* rec = reinterpret_cast<const float4*>(st.buf);
	const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(st.buf + 2048u * ntmax);
	const uint32_t* vids = hdrs + kLanes;
	const uint32_t* slots = vids + kLanes * nvmax;
	const uint32_t hdr = hdrs[lane];
	const uint32_t nv = CUBE ? 8u : (hdr & 15u), nt = CUBE ? 6u : ((hdr >> 4) & 15u);
	bool live = (hdr & 15u) != 0;
	uint32_t vid[NV], last = 0;
	float4 O[NV], D[NV];
	if (live) {
		const Mat mat = load_mat(C.bodies, hdr >> 16);
		live = mat.nvol >= k;
		if (finish && mat.nvol == k) last = __ldg(C.lastmask + (size_t)chunk * kLanes + lane);
		if (live) {
#pragma unroll
			for (uint32_t s = 0; s < NV; s++) {
				if (s < nv) {
					vid[s] = vids[s * kLanes + lane];
					vs.ld2(C, vid[s], O[s], D[s]);
				}
			}
			if constexpr (CUBE) {
				turn_cube(O, D, [&](int t, const float4* Ot, float4* Dt) {
					volume_tet(mat, cluster_rec(rec + lane, t), inv_dt2, Ot, Dt);
				});
			} else {
#pragma unroll 1
				for (uint32_t t = 0; t < nt; t++) {
					const uint32_t sl = slots[t * kLanes + lane];
					float4 Ot[4], Dt[4];
#pragma unroll
					for (int j = 0; j < 4; j++) {
						Ot[j] = O[(sl >> (4 * j)) & 15u];
						Dt[j] = D[(sl >> (4 * j)) & 15u];
					}
					volume_tet(mat, cluster_rec(rec + lane, (int)t), inv_dt2, Ot, Dt);
#pragma unroll
					for (int j = 0; j < 4; j++) D[(sl >> (4 * j)) & 15u] = Dt[j];
				}
			}
		}
	}
	if (next >= 0) stage_issue(C, st, (uint32_t)next, lane);  // records consumed: prefetch
	if (live) {
#pragma unroll
		for (uint32_t s = 0; s < NV; s++) {
			if (s < nv) {
				if (last & (1u << s)) {
					finalize_vertex(C, vid[s], O[s], D[s], inv_dt);
					vs.st_o(C, vid[s], O[s]);
				}
				vs.st_d(C, vid[s], D[s]);
			}
		}
	}
}

template <class VS>
__device__ __forceinline__ void run_vol_chunk(const DevCtx& C, const VS& vs, Stage& st, uint32_t chunk, int next, uint32_t lane,
                                              float inv_dt, float inv_dt2, uint32_t k, bool finish) {
	const uint4 m = st.meta;
	const uint32_t ntmax = m.z & 0xffu, nvmax = (m.z >> 8) & 0xffu;
	if (m.z & kShapeCube)
		vol_chunk<true>(C, vs, st, chunk, ntmax, nvmax, next, lane, inv_dt, inv_dt2, k, finish);
	else
		vol_chunk<false>(C, vs, st, chunk, ntmax, nvmax, next, lane, inv_dt, inv_dt2, k, finish);
}

// One damping pass over a resident chunk (KIND 0: element Rayleigh damping,
// 1: PBD damping); lane = cluster, tets in the cluster's order. The state is
// the canonical (X, V): each vertex's last solve of the substep finished it.
// Only velocities change. CUBE: canonical cube chunks, all in registers. Not
// inlined: the damping passes then cost the solve path no registers.
template <bool CUBE, int KIND, class VS>
__device__ __noinline__ void damp_chunk(const DevCtx& C, const VS& vs, Stage& st, uint32_t ntmax, uint32_t nvmax, uint32_t trow,
                                        int next, uint32_t lane, float inv_dt, uint32_t tick) {
	constexpr uint32_t NV = CUBE ? 8u : kMaxClusterVerts;
	constexpr uint32_t NT = CUBE ? 6u : kMaxClusterTets;
	const float4* rec = reinterpret_cast<const float4*>(st.buf);
	const uint32_t* hdrs = reinterpret_cast<const uint32_t*>(st.buf + 2048u * ntmax);
	const uint32_t* vids = hdrs + kLanes;
	const uint32_t* slots = vids + kLanes * nvmax;
	const uint32_t hdr = hdrs[lane];
	const bool live = (hdr & 15u) != 0;
	const uint32_t nv = CUBE ? 8u : (hdr & 15u), nt = CUBE ? 6u : ((hdr >> 4) & 15u);
	uint32_t vid[NV], some = 0;  // bit t: tet t of the cluster is damped
	float4 X[NV], V[NV];
	if (live) {
		const DampBody d = damp_of(C.bodies[hdr >> 16], tick, KIND);
		const Mat mat = load_mat(C.bodies, hdr >> 16);
		float ar = 0.0f;  // PBD: the area of the tet that is next
		auto on = [&](uint32_t t) {
			const uint32_t f = d.amort ? __ldg(C.tflat + (size_t)(trow + t) * kLanes + lane) : 0u;
			return !d.amort || (f >= d.lo && f < d.hi);
		};
		auto load = [&]() {
#pragma unroll
			for (uint32_t k = 0; k < NV; k++) {
				if (k < nv) {
					vid[k] = vids[k * kLanes + lane];
					vs.ld2(C, vid[k], X[k], V[k]);
				}
			}
		};
		auto damp = [&](int t, const float4* Xt, float4* Vt, float ar) {
			if (KIND == 0)
				rayleigh_tet(mat, cluster_rec(rec + lane, t), Xt, Vt, inv_dt, d.rayleigh);
			else
				pbd_tet(Xt, Vt, fminf(1.0f, d.pbd / ar));
		};
		if constexpr (CUBE) {
			if (d.on) {
				// every tet's place in the order at once
				if (KIND == 1) ar = __ldg(C.tarea + (size_t)trow * kLanes + lane);
#pragma unroll
				for (uint32_t t = 0; t < NT; t++)
					if (on(t)) some |= 1u << t;
			}
			if (some) {
				load();
				// Six tets unrolled were fetched anew for every damping pass: with the
				// solve above, a damped substep of 6,144 tets took 70 us, now 62.
				turn_cube(X, V, [&](int t, const float4* Xt, float4* Vt) {
					const float a = ar;
					if (KIND == 1 && t < 5) ar = __ldg(C.tarea + (size_t)(trow + t + 1) * kLanes + lane);
					if (some >> t & 1u) damp(t, Xt, Vt, a);
				});
			}
		} else if (d.on) {
			// each tet's place and area when its turn comes: collected before the vertices,
			// as for cubes, they cost the grid 1 to 3% (64 x 24 x 16 shuffled, 128 threads, a
			// frame 18,250 -> 17,990 us, mirrored 24,560 -> 24,270)
			some = 1u;
			load();
#pragma unroll 1
			for (uint32_t t = 0; t < nt; t++) {
				if (on(t)) {
					const uint32_t sl = slots[t * kLanes + lane];
					float4 Xt[4], Vt[4];
#pragma unroll
					for (int k = 0; k < 4; k++) {
						Xt[k] = X[(sl >> (4 * k)) & 15u];
						Vt[k] = V[(sl >> (4 * k)) & 15u];
					}
					damp((int)t, Xt, Vt, KIND == 1 ? __ldg(C.tarea + (size_t)(trow + t) * kLanes + lane) : 0.0f);
#pragma unroll
					for (int k = 0; k < 4; k++) V[(sl >> (4 * k)) & 15u] = Vt[k];
				}
			}
		}
	}
	if (next >= 0) stage_issue(C, st, (uint32_t)next, lane);  // records consumed: prefetch
	if (some) {
#pragma unroll
		for (uint32_t k = 0; k < NV; k++) {
			if (k < nv) vs.st_d(C, vid[k], V[k]);
		}
	}
}

// kind 0: element Rayleigh damping, 1: PBD damping.
template <class VS>
__device__ __forceinline__ void run_damp_chunk(const DevCtx& C, const VS& vs, Stage& st, int next, uint32_t lane,
                                               int kind, float inv_dt, uint32_t tick) {
	const uint4 m = st.meta;
	const uint32_t ntmax = m.z & 0xffu, nvmax = (m.z >> 8) & 0xffu, trow = m.w;
	if (m.z & kShapeCube) {
		if (kind == 0)
			damp_chunk<true, 0>(C, vs, st, ntmax, nvmax, trow, next, lane, inv_dt, tick);
		else
			damp_chunk<true, 1>(C, vs, st, ntmax, nvmax, trow, next, lane, inv_dt, tick);
	} else {
		if (kind == 0)
			damp_chunk<false, 0>(C, vs, st, ntmax, nvmax, trow, next, lane, inv_dt, tick);
		else
			damp_chunk<false, 1>(C, vs, st, ntmax, nvmax, trow, next, lane, inv_dt, tick);
	}
}

// Whether damping pass (kind index k >= 1, colour c) has work at this tick.
__device__ __forceinline__ bool pass_on(const DevCtx& C, int dk, uint32_t c, uint32_t tick) {
	return __ldg(C.pass_on + ((size_t)dk * 8u + tick % 8u) * C.ncolours + c) != 0;
}

// Vertices in no tet: nothing else touches them, so one thread takes each
// through all nsub substeps at once (predict, then finalize + predict); the
// final finalize pass closes the last one.
// With damping sweeps the launch ends in the canonical state without a
// closing finalize pass, so these vertices are finalized here (finalize_end).
template <bool TAPE = false, class VS>
__device__ __forceinline__ void run_isolated(const DevCtx& C, const VS& vs, uint32_t begin, uint32_t step, uint32_t nsub, float dt,
                                             float inv_dt, bool finalize_end = false) {
	for (uint32_t i = begin; i < C.nisolated; i += step) {
		const uint32_t v = __ldg(C.isolated + i);
		float4 O, D;
		vs.ld(C, v, O, D);
		for (uint32_t s = 0; s < nsub; s++) {
			const float4 Dbefore = D;
			advance_vertex(C, v, O, D, s == 0, dt, inv_dt);
			if (TAPE) tape_vertex(C, v, O, Dbefore, s, tip_at(C, v, s == 0));
		}
		if (finalize_end) finalize_vertex(C, v, O, D, inv_dt);
		vs.st(C, v, O, D);
	}
}

// Vertices [begin, end) by `step`, read where vs has them, written to vert.
template <bool TAPE = false, class VS>
__device__ __forceinline__ void run_finalize(const DevCtx& C, const VS& vs, uint32_t begin, uint32_t end, uint32_t step,
                                             float inv_dt, uint32_t nsub = 0) {
	for (uint32_t v = begin; v < end; v += step) {
		float4 O, D;
		vs.ld(C, v, O, D);
		if (TAPE) __stcs(C.tape_fin + v, D);
		finalize_vertex(C, v, O, D, inv_dt);
		if (TAPE) {
			const int q = __ldg(C.tip_of + v);
			if (q >= 0) C.traj[(size_t)(C.sub_base + nsub - 1) * C.ntips + q] = O;
		}
		st_vertex(C.vert + 2 * (size_t)v, O, D);
	}
}

// A substep is P = kinds x ncolours passes: the solve sweep over the colours,
// the volume sweeps (DevCtx::nvol), then each damping sweep
// (DevCtx::damp_kinds) over them again; pass q works on colour q % ncolours.
__device__ __forceinline__ uint32_t pass_kinds(const DevCtx& C) {
	return 1u + C.nvol + (uint32_t)__popc(C.damp_kinds);
}

// Damping kind of pass-kind index k > nvol: 0 element Rayleigh, 1 PBD.
__device__ __forceinline__ int damp_kind(const DevCtx& C, uint32_t k) {
	return (k == C.nvol + 1u && (C.damp_kinds & 1u)) ? 0 : 1;
}

// Whether pass q (P passes per substep) runs at `tick`: the solve and volume
// passes always, a damping pass only if some tet of its colour is damped then.
__device__ __forceinline__ bool pass_runs(const DevCtx& C, uint32_t q, uint32_t tick) {
	const uint32_t kind = q / C.ncolours;
	return kind <= C.nvol || pass_on(C, damp_kind(C, kind), q - kind * C.ncolours, tick);
}

// ---- bricks: what the plain and the extended brick kernel share -------------------
__device__ __forceinline__ float4 ld_any(const float4* p) {
	float4 v;
	asm volatile("ld.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ void st_any(float4* p, const float4& v) {
	asm volatile("st.cg.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// A brick chunk's vertex words: a device vertex, or kPrivate | the slot of the
// block's shared memory (O at sv[p], D at sv[pmax + p], device id spid[p]).
// GENERIC: one access through a generic address, past L1, for both, so that a
// warp whose lanes have both takes no branch per vertex; else a branch. With one
// brick per SM the former is faster (a batch of 96 uneven bodies: 3,695 us per four
// frames against 3,815), with two bricks per SM the latter (1,572,864 tets: 902 us
// per frame against 1,073).
template <bool GENERIC>
struct BrickVerts {
	float4* sv;
	const uint32_t* spid;
	uint32_t pmax;

	__device__ __forceinline__ float4* o(const DevCtx& C, uint32_t w) const {
		return (w & kPrivate) ? sv + (w & ~kPrivate) : C.vert + 2 * (size_t)w;
	}
	__device__ __forceinline__ float4* d(const DevCtx& C, uint32_t w) const {
		return (w & kPrivate) ? sv + pmax + (w & ~kPrivate) : C.vert + 2 * (size_t)w + 1;
	}
	__device__ __forceinline__ void ld(const DevCtx& C, uint32_t w, float4& O, float4& D) const {
		if (GENERIC) {
			O = ld_any(o(C, w));
			D = ld_any(d(C, w));
		} else if (w & kPrivate) {
			O = sv[w & ~kPrivate];
			D = sv[pmax + (w & ~kPrivate)];
		} else {
			ld_vertex(C.vert + 2 * (size_t)w, O, D);
		}
	}
	// o_too: O changed as well
	__device__ __forceinline__ void st(const DevCtx& C, uint32_t w, const float4& O, const float4& D, bool o_too) const {
		if (GENERIC) {
			if (o_too) st_any(o(C, w), O);
			st_any(d(C, w), D);
		} else if (w & kPrivate) {
			if (o_too) sv[w & ~kPrivate] = O;
			sv[pmax + (w & ~kPrivate)] = D;
		} else if (o_too) {
			st_vertex(C.vert + 2 * (size_t)w, O, D);
		} else {
			__stcg(C.vert + 2 * (size_t)w + 1, D);
		}
	}
	__device__ __forceinline__ uint32_t id(uint32_t w) const { return (w & kPrivate) ? spid[w & ~kPrivate] : w; }
};

__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
	asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The calling warp's brick chunk buffer and mbarrier.
__device__ __forceinline__ Stage brick_stage_init(uint32_t lane) {
	extern __shared__ __align__(128) uint8_t smem[];
	__shared__ uint64_t bmbars[32];
	const uint32_t w = threadIdx.x >> 5;
	Stage st = {smem + (size_t)w * kBrickChunkBytes, nullptr, &bmbars[w], 0u, -1, make_uint4(0u, 0u, 0u, 0u)};
	if (lane == 0) mbar_init(st.mbar);
	__syncwarp();
	return st;
}

__device__ __forceinline__ void brick_issue(const DevCtx& C, Stage& st, uint32_t chunk, uint32_t lane) {
	__syncwarp();
	if (lane == 0)
		bulk_copy_g2s(st.buf, C.bcblk + (size_t)chunk * (kBrickChunkBytes / 16u), kBrickChunkBytes, st.mbar);
	st.inflight = (int)chunk;
}

// Makes brick chunk `chunk` resident in the warp's buffer; false on timeout.
__device__ __forceinline__ bool brick_acquire(const DevCtx& C, Stage& st, uint32_t chunk, uint32_t lane) {
	if (st.inflight != (int)chunk) {
		if (st.inflight >= 0) {
			if (!mbar_wait(C, st.mbar, st.parity)) return false;
			st.parity ^= 1u;
		}
		brick_issue(C, st, chunk, lane);
	}
	const bool ok = mbar_wait(C, st.mbar, st.parity);
	st.parity ^= 1u;
	st.inflight = -1;
	return ok;
}

// What a lane needs of its resident brick chunk before its vertices. With one brick
// per SM it is read ahead of the wait for the neighbours (a damped frame of 608,256
// tets: 1,418 -> 1,396 us; with two per SM after it: 2,510 us against 2,525 for
// 3,145,728).
struct BrickLane {
	uint32_t hdr, vw[8];
};

__device__ __forceinline__ BrickLane brick_lane(const Stage& st, uint32_t lane) {
	const uint32_t* p = reinterpret_cast<const uint32_t*>(st.buf + 2048u * 6u) + lane;
	BrickLane l;
	l.hdr = p[0];
#pragma unroll
	for (int s = 0; s < 8; s++) l.vw[s] = p[(s + 1) * kLanes];
	return l;
}

// Bounded wait, by the calling threads (`first` of them striding by
// `stride`), until every brick of list[nb0, nb1) (ALL: every brick in [nb0,
// nb1), without a list) has published at least
// `target` passes. Returns false when a wait ran out or another
// block reported an error. The polls are relaxed loads and one acquire
// fence follows them (the acquire pattern of the PTX memory model): an
// acquire load on every poll, or an acquire-release fence, made the
// throughput frame 1.7% and 11% slower.
template <bool ALL = false>
__device__ bool brick_wait(const DevCtx& C, const uint32_t* list, uint32_t nb0, uint32_t nb1, uint32_t target,
                           uint32_t first, uint32_t stride) {
	target += C.wait_miss;
	bool bad = false;
	for (uint32_t i = nb0 + first; i < nb1 && !bad; i += stride) {
		const uint32_t* f = C.bflag + (size_t)(ALL ? i : __ldg(list + i)) * kBrickFlagStride;
		uint32_t spins = 0;
		uint64_t t0 = 0;
		while ((int32_t)(ld_relaxed_gpu(f) - target) < 0) {
			if (++spins == 256) {
				spins = 0;
				if (*(volatile int*)C.err) {
					bad = true;
					break;
				}
				const uint64_t t = global_ns();
				if (t0 == 0) {
					t0 = t;
				} else if (t - t0 > C.timeout_ns) {
					atomicCAS(C.err, 0, kErrBarrierTimeout);
					bad = true;
					break;
				}
			}
		}
	}
	asm volatile("fence.acquire.gpu;" ::: "memory");
	return !bad;
}

}  // namespace

}  // namespace xfem
