// CUDA kernels of libxfem.so (sm_103a): the coloured Gauss-Seidel XPBD substep.
//
// Data layout in HBM (all device-order, see xfem_internal.h):
//   vert[2v]   = (O.x, O.y, O.z, w)   position at the start of the substep and
//                                     inverse mass; between calls: X
//   vert[2v+1] = (D.x, D.y, D.z, bits) displacement within the substep; between
//                                     calls: V. bits = lock | contact | body<<8
// One 32-byte sector per vertex, so a gather touches one sector.
//
// Work unit: a cluster = up to 8 tets sharing vertices, solved in sequence by
// one thread with its (<= 8) vertices staged in shared memory. Clusters of one
// colour share no vertex, so there is no atomic and no race. 32 clusters of a
// colour form a chunk (one warp); chunk data is stored lane-minor so every
// per-lane load of a warp is one contiguous 128- or 512-byte run.
//
// Substep schedule (Geo3d::Substep, XPBDFEM/Geo.cpp:305-356, restated):
//   each colour pass: every cluster first advances the vertices it owns (it is
//              the lowest-colour cluster touching them): finalize the
//              previous substep (locks, ground, V = D/dt, O += D) and predict
//              this one (V += g dt, V *= 1 - drag, D = V dt); then it solves
//              its tets in sequence
//   end      : finalize the last substep back to (X, V)
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "xfem_chunk.cuh"
#include "xfem_device.cuh"
#include "xfem_internal.h"

namespace xfem {

namespace {

// The warp's next chunk after `ch` (pass q of substep s, P passes per
// substep, tick0 the launch's first tick): the next chunk of the same colour,
// else its first chunk of the following passes that run (wrapping into the
// next substep); -1 when the launch has no more work for it.
__device__ __forceinline__ int next_chunk(const DevCtx& C, uint32_t s, uint32_t nsub, uint32_t q, uint32_t P,
                                          uint32_t ch, uint32_t gwarp, uint32_t nwarps, uint32_t tick0 = 0,
                                          const uint32_t* ccb = nullptr) {
	if (!ccb) ccb = C.colour_chunk_begin;
	if (ch + nwarps < ccb[q % C.ncolours + 1]) return (int)(ch + nwarps);
	for (uint32_t k = 1; k <= P; k++) {
		uint32_t q2 = q + k, s2 = s;
		if (q2 >= P) {
			q2 -= P;
			s2++;
		}
		if (s2 >= nsub) return -1;
		if (P > C.ncolours && !pass_runs(C, q2, tick0 + s2)) continue;
		const uint32_t c2 = q2 % C.ncolours;
		const uint32_t first = ccb[c2] + gwarp;
		if (first < ccb[c2 + 1]) return (int)first;
	}
	return -1;
}

// Persistent kernel: nsub substeps x P passes separated by the bounded grid
// barrier. Must be launched cooperatively (co-resident grid). Without damping
// the substep state stays (O, D) between substeps and the closing pass
// finalizes it; with damping sweeps they finish every substep and the state
// between substeps is canonical (X, V).
// EXT: the extended kernel, with the damping sweeps, the in-solve damping,
// the Pixar and cube models and the volume sweeps compiled in (handles that
// use any of them); without it they cost the kernel nothing.
template <bool LAMBDAS, bool TAPE = false, bool EXT = false>
__global__ void __launch_bounds__(256) k_persistent(DevCtx C, uint32_t nsub, float dt) {
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	// chunk i of a colour goes to block i % grid, so chunks spread over all SMs
	const uint32_t gwarp = wib * gridDim.x + blockIdx.x, nwarps = wpb * gridDim.x;
	const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
	const bool dmode = EXT && C.damp_kinds != 0u;
	const uint32_t P = (EXT ? pass_kinds(C) : 1u) * C.ncolours;
	const uint32_t tick0 = __ldcg(C.tick);  // read before the first barrier; block 0 advances it at the end
	Stage st = stage_init(C, lane);
	// the colour table in shared memory (up to 64 colours): read after every
	// barrier, a global load there would sit on each pass's critical path
	__shared__ uint32_t s_ccb[65];
	const bool ccb_sh = C.ncolours <= 64u;
	if (ccb_sh)
		for (uint32_t i = threadIdx.x; i <= C.ncolours; i += blockDim.x) s_ccb[i] = __ldg(C.colour_chunk_begin + i);
	__syncthreads();
	const uint32_t* ccb = ccb_sh ? s_ccb : C.colour_chunk_begin;
	run_isolated<TAPE>(C, GlobalVerts{}, gtid, nthreads, nsub, dt, inv_dt, dmode);
	uint32_t target = C.bar_base;
	bool ok = true;
	for (uint32_t s = 0; s < nsub && ok; s++) {
		for (uint32_t q = 0; q < P && ok; q++) {
			const uint32_t kind = q / C.ncolours, c = q - kind * C.ncolours;
			// a damping pass with nothing to damp at this tick is skipped by
			// every block alike (same table, same tick): no work, no barrier
			if (EXT && kind > 0 && !pass_runs(C, q, tick0 + s)) continue;
			const uint32_t cb = ccb[c], ce = ccb[c + 1];
			for (uint32_t ch = cb + gwarp; ch < ce; ch += nwarps) {
				if (!stage_acquire(C, st, ch, lane)) {
					ok = false;
					break;
				}
				const int next = next_chunk(C, s, nsub, q, P, ch, gwarp, nwarps, tick0, ccb);
				if (!EXT || kind == 0)
					run_chunk<LAMBDAS, TAPE, EXT>(C, GlobalVerts{}, AnyBody{}, st, ch, next, lane, dmode || s == 0, dt, inv_dt, inv_dt2, s,
					                               dmode);
				else if (kind <= C.nvol)
					run_vol_chunk(C, GlobalVerts{}, st, ch, next, lane, inv_dt, inv_dt2, kind, dmode);
				else
					run_damp_chunk(C, GlobalVerts{}, st, next, lane, damp_kind(C, kind), inv_dt, tick0 + s);
			}
			if (!grid_sync(C, target)) ok = false;
		}
	}
	if (!ok) {
		// leave no copy in flight
		if (st.inflight >= 0) mbar_wait(C, st.mbar, st.parity);
		return;
	}
	if (!dmode) run_finalize<TAPE>(C, GlobalVerts{}, gtid, C.nverts, nthreads, inv_dt, nsub);
	if (gtid == 0) *C.tick = tick0 + nsub;
}

// Bounded wait until every neighbour chunk of `ch` has done its share of
// substep s: chunks of a lower colour must have completed s + 1 substeps,
// chunks of a higher colour s substeps (the previous one). One lane per
// neighbour; false (and the error word set) on timeout.
__device__ bool wait_deps(const DevCtx& C, uint32_t ch, uint32_t s, uint32_t lane) {
	const uint32_t b = __ldg(C.dep_begin + ch), e = __ldg(C.dep_begin + ch + 1);
	bool ok = true;
	for (uint32_t i = b + lane; i < e && ok; i += kLanes) {
		const uint32_t d = __ldg(C.deps + i);
		const uint32_t need = s + (d >> 31) + C.wait_miss;
		if (need == 0) continue;
		const uint32_t* f = C.done + (d & 0x7fffffffu);
		uint32_t spins = 0;
		uint64_t t0 = 0;
		while (ld_acquire_gpu(f) < need) {
			if (++spins == 64) {
				spins = 0;
				if (*(volatile int*)C.err) {
					ok = false;
					break;
				}
				const uint64_t t = global_ns();
				if (t0 == 0) {
					t0 = t;
				} else if (t - t0 > C.timeout_ns) {
					atomicCAS(C.err, 0, kErrDepTimeout);
					ok = false;
					break;
				}
			}
		}
	}
	return __all_sync(0xffffffffu, ok);
}

// Persistent dataflow kernel: the same chunk sequence per warp as
// k_persistent, but a chunk waits only for the neighbouring chunks it shares
// vertices with (per-chunk completion counters) instead of a grid barrier per
// colour. Every dependency points to an earlier (substep, colour) item and each
// warp walks its items in that order, so with a co-resident grid the earliest
// unfinished item can always run: no deadlock. One grid barrier ends the
// launch before the final finalize pass.
template <bool LAMBDAS>
__global__ void __launch_bounds__(256) k_dataflow(DevCtx C, uint32_t nsub, float dt) {
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	const uint32_t gwarp = wib * gridDim.x + blockIdx.x, nwarps = wpb * gridDim.x;
	const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
	const uint32_t tick0 = __ldcg(C.tick);
	Stage st = stage_init(C, lane);
	run_isolated(C, GlobalVerts{}, gtid, nthreads, nsub, dt, inv_dt);
	bool ok = true;
	for (uint32_t s = 0; s < nsub && ok; s++) {
		for (uint32_t c = 0; c < C.ncolours && ok; c++) {
			const uint32_t cb = __ldg(C.colour_chunk_begin + c), ce = __ldg(C.colour_chunk_begin + c + 1);
			for (uint32_t ch = cb + gwarp; ch < ce; ch += nwarps) {
				const int next = next_chunk(C, s, nsub, c, C.ncolours, ch, gwarp, nwarps);
				if (st.inflight != (int)ch) stage_issue_or_wait(C, st, ch, lane);  // records do not depend on neighbours
				if (!wait_deps(C, ch, s, lane) || !stage_acquire(C, st, ch, lane)) {
					ok = false;
					break;
				}
				run_chunk<LAMBDAS>(C, GlobalVerts{}, AnyBody{}, st, ch, next, lane, s == 0, dt, inv_dt, inv_dt2);
				__syncwarp();
				if (lane == 0) {
					__threadfence();
					st_release_gpu(C.done + ch, s + 1);
				}
			}
		}
	}
	if (!ok && st.inflight >= 0) {
		mbar_wait(C, st.mbar, st.parity);  // leave no copy in flight
		st.inflight = -1;
	}
	uint32_t target = C.bar_base;
	if (!grid_sync(C, target) || !ok) return;
	run_finalize(C, GlobalVerts{}, gtid, C.nverts, nthreads, inv_dt);
	if (gtid == 0) *C.tick = tick0 + nsub;
}

// ---- brick launch form (sync_mode 4) ------------------------------------------
//
// The clusters are split into spatially compact bricks, one per block. A
// vertex that only one brick's clusters touch stays in that block's shared
// memory for the whole launch; the others stay in vert (L2). A pass is the
// brick's chunks of one colour; instead of a grid barrier the block then
// publishes its pass count and waits for the bricks it shares vertices with.
// Any vertex a pass reads was last written by a brick that shares it, which
// has finished the previous pass; no brick can be more than one pass ahead of
// a brick it shares vertices with. The colour order, the clusters and the
// arithmetic are those of k_persistent, so the results are bit-identical.

// The warp's next brick chunk after `ch` (colour c of substep s; bcb: the
// brick's colour chunk offsets), -1 when the launch has no more for it.
__device__ __forceinline__ int next_brick_chunk(const uint32_t* bcb, uint32_t ncol, uint32_t s, uint32_t nsub,
                                                uint32_t c, uint32_t ch, uint32_t wib, uint32_t wpb) {
	if (ch + wpb < bcb[c + 1]) return (int)(ch + wpb);
	for (uint32_t k = 1; k <= ncol; k++) {
		uint32_t c2 = c + k, s2 = s;
		if (c2 >= ncol) {
			c2 -= ncol;
			s2++;
		}
		if (s2 >= nsub) return -1;
		const uint32_t f = bcb[c2] + wib;
		if (f < bcb[c2 + 1]) return (int)f;
	}
	return -1;
}

// One resident brick chunk (every lane a whole cube, as run_chunk_cube).
// Its vertex words are BrickVerts'; a brick's O and D are two arrays so that the
// 16-byte accesses of a warp, whose lanes hold nearby slots, fall in different
// bank groups.
// bodies: the body parameters (a shared-memory copy when the handle has few).
// ONE: a single body, whose parameters bp1 and material mat1 the kernel holds
// in registers.
template <bool ONE, bool PAIR, bool GENERIC>
__device__ __forceinline__ void run_chunk_brick(const DevCtx& C, Stage& st, const BrickLane& bl, int next, uint32_t lane, bool first,
                                                float dt, float inv_dt, float inv_dt2, const BrickVerts<GENERIC>& vs,
                                                const BodyParams* bodies, bool bshared,
                                                const BodyParams& bp1, const Mat& mat1) {
	const float4* rec = reinterpret_cast<const float4*>(st.buf);
	const uint32_t hdr = bl.hdr;
	const uint32_t* vw = bl.vw;
	const bool live = (hdr & 15u) != 0;
	const uint32_t mask = (hdr >> 8) & 0xffu;
	float4 O[8], D[8];
	if (live) {
		const Mat mat = ONE ? mat1 : bshared ? load_mat_shared(bodies, hdr >> 16) : load_mat(bodies, hdr >> 16);
#pragma unroll
		for (int s = 0; s < 8; s++) vs.ld(C, vw[s], O[s], D[s]);
#pragma unroll
		for (int s = 0; s < 8; s++)
			if (mask & (1u << s)) {
				const uint32_t v = vs.id(vw[s]);
				if (ONE)
					advance_vertex_bp(C, bp1, v, O[s], D[s], first, dt, inv_dt);
				else
					advance_vertex(C, v, O[s], D[s], first, dt, inv_dt, bodies);
			}
		solve_cube<false, !PAIR>(
		    mat, rec + lane, inv_dt, inv_dt2, O, D, [](int, const float4*) {}, [](int, const float2&) {});
	}
	if (next >= 0) brick_issue(C, st, (uint32_t)next, lane);  // buffer consumed: prefetch
	if (live) {
#pragma unroll
		for (int s = 0; s < 8; s++) vs.st(C, vw[s], O[s], D[s], (mask & (1u << s)) != 0u);
	}
}

// Persistent brick kernel: one block per brick (grid = nbricks, cooperative
// launch so that every brick is resident), the plain solve only (no damping,
// volume passes or multiplier output). The state between substeps stays
// (O, D), and each brick finalizes its own vertices at the end.
// PAIR: two bricks per SM, of 192 threads at most and so of 168 registers a
// thread. Told that bound, the compiler schedules within it (a frame of 1,572,864
// tets: 928 us before, 902 so; reading records ahead would spill: 939). One brick
// per SM has registers left, and reads a tet's record while the one before is
// solved (four frames of a batch of 96 uneven bodies: 4,086 -> 3,815 us, and 3,695
// with the vertices through generic addresses).
template <bool ONE, bool PAIR, bool GENERIC>
__global__ void __launch_bounds__(PAIR ? 192 : 256, PAIR ? 2 : 1) k_bricks(DevCtx C, uint32_t nsub, float dt) {
	extern __shared__ __align__(128) uint8_t smem[];
	__shared__ uint32_t s_bcb[65], s_bwait[64];
	__shared__ BodyParams s_bodies[kBrickBodies];
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	const uint32_t b = blockIdx.x, ncol = C.ncolours;
	const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
	const uint32_t tick0 = __ldcg(C.tick);  // read before any brick publishes; block 0 advances it at the end
	Stage st = brick_stage_init(lane);
	float4* sv = reinterpret_cast<float4*>(smem + (size_t)wpb * kBrickChunkBytes);
	uint32_t* spid = reinterpret_cast<uint32_t*>(sv + 2 * (size_t)C.bpriv_max);
	const BrickVerts<GENERIC> vs = {sv, spid, C.bpriv_max};
	for (uint32_t i = threadIdx.x; i <= ncol; i += blockDim.x) {
		s_bcb[i] = __ldg(C.bchunk_begin + (size_t)b * ncol + i);
		if (i < ncol) s_bwait[i] = __ldg(C.bchunk_wait_end + (size_t)b * ncol + i);
	}
	// few bodies: their parameters in shared memory (the advance reads them per vertex)
	const bool bshared = C.nbodies <= kBrickBodies;
	if (bshared) {
		const uint32_t words = C.nbodies * (uint32_t)(sizeof(BodyParams) / 4);
		for (uint32_t i = threadIdx.x; i < words; i += blockDim.x)
			reinterpret_cast<uint32_t*>(s_bodies)[i] = __ldg(reinterpret_cast<const uint32_t*>(C.bodies) + i);
	}
	const BodyParams* bodies = bshared ? s_bodies : C.bodies;
	// a single body: its parameters and material in registers
	BodyParams bp1;
	Mat mat1;
	if (ONE) {
		bp1 = C.bodies[0];
		mat1 = load_mat(C.bodies, 0);
	}
	// the brick's own vertices into shared memory, for the whole launch
	const uint32_t pb = __ldg(C.bpriv_begin + b), pe = __ldg(C.bpriv_begin + b + 1);
	for (uint32_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
		const uint32_t v = __ldg(C.bpriv_vid + i);
		float4 O, D;
		ld_vertex(C.vert + 2 * (size_t)v, O, D);
		sv[i - pb] = O;
		sv[C.bpriv_max + (i - pb)] = D;
		spid[i - pb] = v;
	}
	__syncthreads();
	// vertices in no tet, finalized here too (no closing pass over all vertices)
	run_isolated(C, GlobalVerts{}, gtid, nthreads, nsub, dt, inv_dt, true);
	const uint32_t nb0 = __ldg(C.bnb_begin + b), nb1 = __ldg(C.bnb_begin + b + 1);
	// A pass: the warps whose chunk holds only interior clusters (every vertex
	// private) start at once; a warp with a boundary cluster first waits
	// until the neighbouring bricks have finished the previous pass (their
	// writes to the shared vertices are visible). The block's barrier then
	// ends the pass, and it publishes the pass count. The chain over the bricks is a
	// boundary warp's work (6,700 to 7,700 cycles), the publication (1,700) and the
	// wait's last poll; the chunk's copy and the choice of the next one come before
	// the wait (after it they cost 500: 912 -> 887 us per frame of 1,572,864 tets).
	uint32_t epoch = 0;
	bool ok = true;
	for (uint32_t s = 0; s < nsub && ok; s++) {
		for (uint32_t c = 0; c < ncol && ok; c++) {
			const uint32_t wend = s_bwait[c];
			bool bad = false, waited = false;
			for (uint32_t ch = s_bcb[c] + wib; ch < s_bcb[c + 1] && !bad; ch += wpb) {
				if (!brick_acquire(C, st, ch, lane)) {
					bad = true;
					break;
				}
				const int next = next_brick_chunk(s_bcb, ncol, s, nsub, c, ch, wib, wpb);
				BrickLane bl;
				if (!PAIR) bl = brick_lane(st, lane);
				if (ch < wend && !waited) {
					const uint32_t q = b * ncol + c;
					bad = __any_sync(0xffffffffu, !brick_wait(C, C.bcnb, __ldg(C.bcnb_begin + q),
					                                             __ldg(C.bcnb_begin + q + 1), epoch, lane, 32u));
					__syncwarp();  // orders every lane's loads after the lanes' acquires
					waited = true;
					if (bad) break;
				}
				if (PAIR) bl = brick_lane(st, lane);
				run_chunk_brick<ONE, PAIR, GENERIC>(C, st, bl, next, lane, s == 0, dt, inv_dt, inv_dt2, vs, bodies, bshared, bp1,
				                     mat1);
			}
			if (__syncthreads_or(bad ? 1 : 0)) {
				ok = false;
				break;
			}
			++epoch;
			// the release store orders every write of the pass that the
			// barrier made visible to this thread before the count
			if (threadIdx.x == 0) st_release_gpu(C.bflag + (size_t)b * kBrickFlagStride, epoch);
		}
	}
	// every brick sharing a vertex with this one has finished the last pass
	if (ok) ok = !__syncthreads_or(brick_wait(C, C.bnb, nb0, nb1, epoch, threadIdx.x, blockDim.x) ? 0 : 1);
	if (!ok) {
		if (st.inflight >= 0) mbar_wait(C, st.mbar, st.parity);  // leave no copy in flight
		return;
	}
	for (uint32_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
		const uint32_t v = __ldg(C.bpriv_vid + i);
		float4 O = sv[i - pb], D = sv[C.bpriv_max + (i - pb)];
		if (ONE)
			finalize_vertex_bp(C, bp1, v, O, D, inv_dt);
		else
			finalize_vertex(C, v, O, D, inv_dt, bodies);
		st_vertex(C.vert + 2 * (size_t)v, O, D);
	}
	const uint32_t fb = __ldg(C.bfin_begin + b), fe = __ldg(C.bfin_begin + b + 1);
	for (uint32_t i = fb + threadIdx.x; i < fe; i += blockDim.x) {
		const uint32_t v = __ldg(C.bfin_vid + i);
		float4 O, D;
		ld_vertex(C.vert + 2 * (size_t)v, O, D);
		if (ONE)
			finalize_vertex_bp(C, bp1, v, O, D, inv_dt);
		else
			finalize_vertex(C, v, O, D, inv_dt, bodies);
		st_vertex(C.vert + 2 * (size_t)v, O, D);
	}
	if (gtid == 0) *C.tick = tick0 + nsub;
}

// One colour pass as its own launch (CUDA-graph mode): one chunk per warp.
// kind 0 is the solve pass (first: the state is canonical), 1..nvol the
// volume passes, the rest the damping passes (damp_kind); sub: the substep's
// index in the call (its tick is *C.tick + sub). In the first launch of a
// call, blocks past the colour's chunks step the isolated vertices through
// all nsub substeps.
template <bool LAMBDAS, bool EXT = false>
__global__ void __launch_bounds__(256, 1) k_colour(DevCtx C, uint32_t colour, int first, float dt, uint32_t solve_blocks,
                                                uint32_t nsub, uint32_t kind, uint32_t sub) {
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	if (blockIdx.x >= solve_blocks) {
		const uint32_t b = blockIdx.x - solve_blocks, nb = gridDim.x - solve_blocks;
		run_isolated(C, GlobalVerts{}, b * blockDim.x + threadIdx.x, nb * blockDim.x, nsub, dt, inv_dt, EXT && C.damp_kinds != 0u);
		return;
	}
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t ch = __ldg(C.colour_chunk_begin + colour) + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
	if (ch >= __ldg(C.colour_chunk_begin + colour + 1)) return;
	const uint32_t tick = __ldcg(C.tick) + sub;
	const bool damp_pass = EXT && kind > C.nvol;
	const int dk = damp_pass ? damp_kind(C, kind) : 0;
	// a graph replays its launches at every tick: a damping pass with nothing
	// to damp at this one returns at once
	if (damp_pass && !pass_on(C, dk, colour, tick)) return;
	Stage st = stage_init(C, lane);
	if (!stage_acquire(C, st, ch, lane)) return;
	const bool dmode = EXT && C.damp_kinds != 0u;
	if (!EXT || kind == 0)
		run_chunk<LAMBDAS, false, EXT>(C, GlobalVerts{}, AnyBody{}, st, ch, -1, lane, first != 0, dt, inv_dt, inv_dt2, 0, dmode);
	else if (!damp_pass)
		run_vol_chunk(C, GlobalVerts{}, st, ch, -1, lane, inv_dt, inv_dt2, kind, dmode);
	else
		run_damp_chunk(C, GlobalVerts{}, st, -1, lane, dk, inv_dt, tick);
}

__global__ void k_finalize(DevCtx C, float dt) {
	run_finalize(C, GlobalVerts{}, blockIdx.x * blockDim.x + threadIdx.x, C.nverts, gridDim.x * blockDim.x, 1.0f / dt);
}

// Advances the tick word by a call's substeps (CUDA-graph mode).
__global__ void k_advance_tick(DevCtx C, uint32_t nsub) { *C.tick += nsub; }

// ---- transfers ----------------------------------------------------------------
// One body's positions (which 0), velocities (1), inverse masses (2) or contact
// bits (3) in caller order, and the handle's error word, into memory of the device
// or the host. The words go through shared memory: stored as each thread has them,
// three words 12 bytes apart, a warp's positions took three partial writes of
// every line of host memory (two reads of 279,825 vertices: 4 us more). The error
// word goes with them: a read of 11,550 vertices took 18 us with a copy of its own
// behind the kernel, and takes 14, most of it the launch and the wait.
__global__ void __launch_bounds__(256) k_gather_xyz(const float4* __restrict__ vert, int which, const uint32_t* __restrict__ dev_of,
                                                    uint32_t n, float* __restrict__ out, const int* __restrict__ err,
                                                    int* __restrict__ err_out) {
	__shared__ __align__(16) float s[768];
	const uint32_t first = blockIdx.x * 256u, i = first + threadIdx.x;
	if (err_out && i == 0) *err_out = *err;
	float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
	if (i < n) a = vert[2 * (size_t)dev_of[i] + (which & 1)];
	if (which >= 2) {
		if (i < n) out[i] = which == 2 ? a.w : (__float_as_uint(a.w) & kFlagContact) ? 1.0f : 0.0f;
		return;
	}
	s[3 * threadIdx.x] = a.x;
	s[3 * threadIdx.x + 1] = a.y;
	s[3 * threadIdx.x + 2] = a.z;
	__syncthreads();
	float* o = out + 3 * (size_t)first;
	const uint32_t words = 3u * min(256u, n - first);
	const uint32_t quads = (reinterpret_cast<uintptr_t>(out) & 15u) ? 0u : words / 4u;  // a block starts 3,072 bytes on
	if (threadIdx.x < quads) reinterpret_cast<float4*>(o)[threadIdx.x] = reinterpret_cast<const float4*>(s)[threadIdx.x];
	for (uint32_t k = 4u * quads + threadIdx.x; k < words; k += 256u) o[k] = s[k];
}

__global__ void k_scatter_xyz(float4* __restrict__ vert, int which, const uint32_t* __restrict__ dev_of, uint32_t n,
                              const float* __restrict__ in) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	float4* p = vert + 2 * (size_t)dev_of[i] + which;
	float4 a = *p;
	a.x = in[3 * (size_t)i];
	a.y = in[3 * (size_t)i + 1];
	a.z = in[3 * (size_t)i + 2];
	*p = a;
}

// Per-tet material change without re-uploading the chunk blocks: the
// record's c0 = (1/mu)/volume, formed with the same two correctly rounded
// divisions as the host (XPBDFEM/Fem.cpp:449), and 1/mu for the adjoint.
__global__ void k_set_c0(float4* __restrict__ cblk, const uint32_t* __restrict__ rec, const float* __restrict__ vol,
                         const float* __restrict__ mu, float mu_uniform, uint32_t n, float* __restrict__ inv_mu) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const float im = 1.0f / (mu ? mu[i] : mu_uniform);
	cblk[rec[i]].w = im / vol[i];
	inv_mu[i] = im;
}

// dL/dmu in caller tet order from the per-row accumulator (-mu dL/dmu).
__global__ void k_gather_dmu(const float* __restrict__ cbar, const uint32_t* __restrict__ slot,
                             const float* __restrict__ inv_mu, uint32_t n, float* __restrict__ out) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	out[i] = -cbar[slot[i]] * inv_mu[i];
}

// CalculateElementVolume for T4 (XPBDFEM/Fem.cpp:1066) summed in double.
__global__ void k_volume(const float4* __restrict__ vert, const uint32_t* __restrict__ tets, uint32_t nt,
                         double* __restrict__ out) {
	__shared__ double red[32];
	double acc = 0.0;
	for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
		const float4 x0 = vert[2 * (size_t)tets[4 * (size_t)t]], x1 = vert[2 * (size_t)tets[4 * (size_t)t + 1]];
		const float4 x2 = vert[2 * (size_t)tets[4 * (size_t)t + 2]], x3 = vert[2 * (size_t)tets[4 * (size_t)t + 3]];
		const double a = (double)x0.x - x3.x, b = (double)x1.x - x3.x, c = (double)x2.x - x3.x;
		const double d = (double)x0.y - x3.y, e = (double)x1.y - x3.y, f = (double)x2.y - x3.y;
		const double g = (double)x0.z - x3.z, h = (double)x1.z - x3.z, i = (double)x2.z - x3.z;
		acc += (a * (e * i - f * h) - b * (d * i - f * g) + c * (d * h - e * g)) / 6.0;
	}
	for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x < 32) {
		acc = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
		for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
		if (threadIdx.x == 0) atomicAdd(out, acc);
	}
}

}  // namespace

size_t solve_smem_bytes(int block, uint32_t warp_smem) { return (size_t)(block / 32) * warp_smem; }

// The dynamic shared-memory limit is a property of the kernel on one device
// (cudaFuncSetAttribute acts in the current device's context), shared by
// every handle on that device: it only ever grows to the largest size any
// handle launches with (a larger limit does not restrict smaller launches),
// so one handle's configuration cannot lower another's below what it needs.
// Kept per (device, kernel); a failed raise is returned and not recorded.
static cudaError_t set_smem_attr(const void* f, size_t bytes) {
	struct Entry {
		int dev;
		const void* f;
		size_t bytes;
	};
	static std::mutex mu;
	static std::vector<Entry> done;
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	std::lock_guard<std::mutex> lk(mu);
	for (auto& d : done)
		if (d.dev == dev && d.f == f) {
			if (bytes > d.bytes) {
				e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
				if (e == cudaSuccess) d.bytes = bytes;
			}
			return e;
		}
	e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
	if (e == cudaSuccess) done.push_back({dev, f, bytes});
	return e;
}

static const void* persistent_fn(bool lambdas, bool ext) {
	if (ext) return lambdas ? (const void*)k_persistent<true, false, true> : (const void*)k_persistent<false, false, true>;
	return lambdas ? (const void*)k_persistent<true> : (const void*)k_persistent<false>;
}

static const void* colour_fn(bool lambdas, bool ext) {
	if (ext) return lambdas ? (const void*)k_colour<true, true> : (const void*)k_colour<false, true>;
	return lambdas ? (const void*)k_colour<true> : (const void*)k_colour<false>;
}

int configure_kernels(const LaunchCfg& cfg) {
	const size_t smem = solve_smem_bytes(cfg.block, cfg.warp_smem);
	cudaError_t e = cudaSuccess;
	for (bool ext : {false, true}) {
		if (e == cudaSuccess) e = set_smem_attr(persistent_fn(cfg.lambdas, ext), smem);
		if (e == cudaSuccess) e = set_smem_attr(colour_fn(cfg.lambdas, ext), smem);
	}
	if (e == cudaSuccess)
		e = set_smem_attr(cfg.lambdas ? (const void*)k_dataflow<true> : (const void*)k_dataflow<false>, smem);
	return (int)e;
}

size_t brick_smem_bytes(int block, uint32_t bpriv_max) {
	return (size_t)(block / 32) * kBrickChunkBytes + (size_t)bpriv_max * kBrickVertexBytes;
}

// GENERIC vertex accesses with one brick per SM, of six chunks of a colour at most, where every
// vertex of one brick only has a slot: the bricks of every handle that leaves their number to
// the library. Larger ones (a number that the caller chose) keep the branch: with more of
// their vertices in vert, one 256-bit access is faster than two generic ones, and a second
// round of chunks hides the branch. Measured, us per frame, generic and branch: 98,304 cubes
// in 152 bricks (2.5 chunks) 651 and 688, in 80 (4.8) 755 and 779, in 50 (7.7) 1,197 and
// 1,173; 262,144 in 152 (6.7) 1,050 and 1,001, in 80 (12.8) 1,768 and 1,480; without slots for
// all, 98,304 in 5 13,310 and 7,080, 737,280 in 152 2,820 and 2,225. Two bricks per SM: the
// branch (BrickVerts).
const void* bricks_fn(bool one, bool pair, bool generic) {
	if (pair) return one ? (const void*)k_bricks<true, true, false> : (const void*)k_bricks<false, true, false>;
	if (generic) return one ? (const void*)k_bricks<true, false, true> : (const void*)k_bricks<false, false, true>;
	return one ? (const void*)k_bricks<true, false, false> : (const void*)k_bricks<false, false, false>;
}

int brick_grid_fits(const DevCtx& ctx, int block, bool* fits) {
	const size_t smem = brick_smem_bytes(block, ctx.bpriv_max);
	int dev = 0, sms = 0, per_sm = 1 << 20;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	for (int one = 0; one < 2 && e == cudaSuccess; one++) {
		const void* f = bricks_fn(one != 0, ctx.nbricks > (uint32_t)sms, ctx.bgeneric != 0u);
		int n = 0;
		e = set_smem_attr(f, smem);
		if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, block, smem);
		per_sm = std::min(per_sm, n);
	}
	if (e != cudaSuccess) return (int)e;
	*fits = (uint64_t)per_sm * (uint64_t)sms >= ctx.nbricks && ctx.nbricks > 0;
	return 0;
}

int persistent_grid(const LaunchCfg& cfg, int* blocks_out) {
	const void* f = cfg.sync_mode == 3
	                    ? (cfg.lambdas ? (const void*)k_dataflow<true> : (const void*)k_dataflow<false>)
	                    : persistent_fn(cfg.lambdas, cfg.ext);
	const size_t smem = solve_smem_bytes(cfg.block, cfg.warp_smem);
	int dev = 0, sms = 0, per_sm = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, cfg.block, smem);
	if (e != cudaSuccess) return (int)e;
	*blocks_out = per_sm * sms;
	return per_sm > 0 ? 0 : (int)cudaErrorInvalidConfiguration;
}

int launch_substeps(const DevCtx& ctx, const LaunchCfg& cfg, uint32_t nsub, float dt, void* stream) {
	cudaStream_t st = (cudaStream_t)stream;
	const size_t smem = solve_smem_bytes(cfg.block, cfg.warp_smem);
	cudaError_t e = cudaSuccess;
	if (nsub == 0) return 0;
	if (cfg.sync_mode == 4) {
		// pass counters start at 0; one launch counts at most 2^30 passes
		const size_t smem_b = brick_smem_bytes(cfg.block, ctx.bpriv_max);
		const uint32_t per = std::max(1u, (1u << 30) / std::max(1u, ctx.ncolours));
		int dev = 0, sms = 0;
		e = cudaGetDevice(&dev);
		if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
		if (e != cudaSuccess) return (int)e;
		for (uint32_t done = 0; done < nsub;) {
			uint32_t n = std::min(per, nsub - done);
			e = cudaMemsetAsync(ctx.bflag, 0, sizeof(uint32_t) * kBrickFlagStride * ctx.nbricks, st);
			if (e != cudaSuccess) return (int)e;
			DevCtx c = ctx;
			float dtv = dt;
			void* args[] = {&c, &n, &dtv};
			const void* f = bricks_fn(ctx.nbodies == 1, ctx.nbricks > (uint32_t)sms, ctx.bgeneric != 0u);
			note_launch(XFEM_FORM_BRICKS, ctx.nbricks, (uint32_t)cfg.block, 1);
			e = cudaLaunchCooperativeKernel(f, dim3(ctx.nbricks), dim3(cfg.block), args, smem_b, st);
			if (e != cudaSuccess) return (int)e;
			done += n;
		}
		return 0;
	}
	if (cfg.sync_mode == 1 && cfg.brick_ext && !ctx.bar_base)
		return launch_bricks_ext(ctx, cfg.block, nsub, dt, stream);
	// the hooks that make grid-barrier waits run out or wrap need that barrier
	if (cfg.sync_mode == 1 && cfg.cluster.blocks && !ctx.wait_miss && !ctx.bar_base)
		return launch_cluster(ctx, cfg.cluster, cfg.block, false, cfg.ext_level(), nsub, dt, stream);
	if (cfg.sync_mode == 1 || cfg.sync_mode == 3) {
		e = reset_barrier(ctx, st);
		if (e == cudaSuccess && cfg.sync_mode == 3) e = cudaMemsetAsync(ctx.done, 0, sizeof(uint32_t) * ctx.nchunks, st);
		if (e != cudaSuccess) return (int)e;
		DevCtx c = ctx;
		void* args[] = {&c, &nsub, &dt};
		const void* f = cfg.sync_mode == 1
		                    ? persistent_fn(cfg.lambdas, cfg.ext)
		                    : (cfg.lambdas ? (const void*)k_dataflow<true> : (const void*)k_dataflow<false>);
		note_launch(cfg.sync_mode == 1 ? XFEM_FORM_GRID : XFEM_FORM_DATAFLOW, (uint32_t)cfg.blocks, (uint32_t)cfg.block, 1);
		e = cudaLaunchCooperativeKernel(f, dim3(cfg.blocks), dim3(cfg.block), args, smem, st);
		return (int)e;
	}
	// per-colour launches (captured into a CUDA graph by the caller when wanted):
	// per substep the solve sweep, the volume sweeps, then each damping sweep
	const void* fc = colour_fn(cfg.lambdas, cfg.ext);
	const uint32_t warps_per_block = cfg.block / 32;
	const bool dmode = cfg.ext && ctx.damp_kinds != 0u;
	const uint32_t kinds = cfg.ext ? 1u + ctx.nvol + (uint32_t)__builtin_popcount(ctx.damp_kinds) : 1u;
	uint32_t largest = 0;
	for (uint32_t s = 0; s < nsub; s++) {
		for (uint32_t kind = 0; kind < kinds; kind++) {
			for (uint32_t c = 0; c < ctx.ncolours; c++) {
				const uint32_t nch = cfg.colour_chunk_begin_host[c + 1] - cfg.colour_chunk_begin_host[c];
				uint32_t sb = (nch + warps_per_block - 1) / warps_per_block;
				uint32_t extra = 0;
				if (s == 0 && kind == 0 && c == 0 && ctx.nisolated) extra = (ctx.nisolated + cfg.block - 1) / cfg.block;
				const uint32_t grid = sb + extra;
				if (grid == 0) continue;
				largest = std::max(largest, grid);
				DevCtx cc = ctx;
				uint32_t colour = c, ns = nsub, kd = kind, sub = s;
				int first = (dmode || s == 0) ? 1 : 0;
				float dtv = dt;
				void* args[] = {&cc, &colour, &first, &dtv, &sb, &ns, &kd, &sub};
				e = cudaLaunchKernel(fc, dim3(grid), dim3(cfg.block), args, smem, st);
				if (e != cudaSuccess) return (int)e;
			}
		}
	}
	note_launch(XFEM_FORM_GRAPH, largest, (uint32_t)cfg.block, 1);
	const uint32_t fb = (ctx.nverts + 255) / 256;
	if (fb && !dmode) {
		k_finalize<<<fb, 256, 0, st>>>(ctx, dt);
		e = cudaGetLastError();
		if (e != cudaSuccess) return (int)e;
	}
	k_advance_tick<<<1, 1, 0, st>>>(ctx, nsub);
	return (int)cudaGetLastError();
}

// The recording forward: k_cluster or, for larger handles, k_persistent with the tape writes compiled in. The
// arithmetic is the same inlined code as the plain launch, so the trajectory
// is the plain launch's bit for bit.
int launch_substeps_tape(const DevCtx& ctx, int block, uint32_t warp_smem, uint32_t max_colour_chunks, uint32_t nsub,
                         float dt, void* stream) {
	if (nsub == 0) return 0;
	cudaStream_t st = (cudaStream_t)stream;
	ClusterPlan plan;
	if (!ctx.wait_miss && !ctx.bar_base) {
		const int ec = cluster_plan(ctx, max_colour_chunks, block, true, 0, &plan);
		if (ec) return ec;
	}
	if (plan.blocks) return launch_cluster(ctx, plan, block, true, 0, nsub, dt, stream);
	const void* f = (const void*)k_persistent<false, true>;
	const size_t smem = solve_smem_bytes(block, warp_smem);
	cudaError_t e = set_smem_attr(f, smem);
	int dev = 0, sms = 0, per_sm = 0;
	if (e == cudaSuccess) e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, block, smem);
	if (e != cudaSuccess) return (int)e;
	if (per_sm <= 0) return (int)cudaErrorInvalidConfiguration;
	e = reset_barrier(ctx, st);
	if (e != cudaSuccess) return (int)e;
	DevCtx c = ctx;
	void* args[] = {&c, &nsub, &dt};
	note_launch(XFEM_FORM_GRID, (uint32_t)(per_sm * sms), (uint32_t)block, 1);
	return (int)cudaLaunchCooperativeKernel(f, dim3(per_sm * sms), dim3(block), args, smem, st);
}

int launch_gather_xyz(const float4* vert, int which, const uint32_t* dev_of_caller, uint32_t n, float* out,
                      const int* err, int* err_out, void* stream) {
	if (!n) return 0;
	k_gather_xyz<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(vert, which, dev_of_caller, n, out, err, err_out);
	return (int)cudaGetLastError();
}

int launch_scatter_xyz(float4* vert, int which, const uint32_t* dev_of_caller, uint32_t n, const float* in,
                       void* stream) {
	if (!n) return 0;
	k_scatter_xyz<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(vert, which, dev_of_caller, n, in);
	return (int)cudaGetLastError();
}

int launch_set_c0(float4* cblk, const uint32_t* rec, const float* vol, const float* mu, float mu_uniform, uint32_t n,
                  float* inv_mu, void* stream) {
	if (!n) return 0;
	k_set_c0<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(cblk, rec, vol, mu, mu_uniform, n, inv_mu);
	return (int)cudaGetLastError();
}

int launch_gather_dmu(const float* cbar, const uint32_t* slot, const float* inv_mu, uint32_t n, float* out,
                      void* stream) {
	if (!n) return 0;
	k_gather_dmu<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(cbar, slot, inv_mu, n, out);
	return (int)cudaGetLastError();
}

int launch_volume(const float4* vert, const uint32_t* tets_dev, uint32_t nt, double* out, void* stream) {
	cudaStream_t st = (cudaStream_t)stream;
	cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), st);
	if (e != cudaSuccess || !nt) return (int)e;
	uint32_t grid = (nt + 255) / 256;
	grid = grid > 1024 ? 1024 : grid;
	k_volume<<<grid, 256, 0, st>>>(vert, tets_dev, nt, out);
	return (int)cudaGetLastError();
}


// ---- allocation-free stepping ---------------------------------------------------
// Some callers cannot allocate device memory at the moment they step: a
// process whose device memory is fully reserved by another allocator (a
// framework's caching pool), or a real-time loop that must not take
// cudaMalloc's implicit device-wide synchronisation. For them the persistent
// substep kernel is launched with its scratch words (the grid-barrier arrival
// counter and the device error word) taken from this fixed array instead of
// buffers of the handle, and without the autotuner or CUDA-graph builder,
// which may allocate.
//
// The array lives in every device that loads the library until the process
// exits. All calls share it and it keeps the last call's contents, so each
// call sets the words it uses first; calls whose kernels overlap on one GPU
// would race on it and must not be issued.
namespace {
constexpr uint32_t kNoAllocScratchWords = 64;  // 256 bytes; words 0 and 1 are used
static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocScratchWords];
constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
uint32_t* g_noalloc_ptr[kNoAllocMaxDevices] = {};
}  // namespace

int launch_substeps_noalloc(const DevCtx& ctx, int block, uint32_t warp_smem, bool lambdas, uint32_t nsub, float dt,
                            void* stream, int device, int* device_error) {
	if (device < 0 || device >= kNoAllocMaxDevices) return (int)cudaErrorInvalidDevice;
	uint32_t* p = nullptr;
	{
		// Set-up, once per device, with that device current: the array's name
		// in host code is a host-side stand-in, so its device address is
		// looked up and passed to the kernel.
		std::lock_guard<std::mutex> lk(g_noalloc_mu);
		if (!g_noalloc_ptr[device]) {
			const cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
			if (e != cudaSuccess) return (int)e;
			g_noalloc_ptr[device] = p;
		}
		p = g_noalloc_ptr[device];
	}
	cudaStream_t st = (cudaStream_t)stream;
	const void* f = persistent_fn(lambdas, ctx.ext != 0u);
	const size_t smem = solve_smem_bytes(block, warp_smem);
	cudaError_t e = set_smem_attr(f, smem);  // no allocation: the kernel's shared-memory limit on this device
	int sms = 0, per_sm = 0;
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, block, smem);
	if (e != cudaSuccess) return (int)e;
	if (per_sm <= 0) return (int)cudaErrorInvalidConfiguration;
	const uint32_t blocks = (uint32_t)(per_sm * sms);
	// One call's grid-barrier arrivals stay below 2^31: every block arrives
	// once per pass, and a substep runs (1 + volume sweeps + damping kinds) x
	// colours passes in the extended kernel, one per colour otherwise.
	const uint64_t kinds = ctx.ext ? 1ull + ctx.nvol + (uint64_t)__builtin_popcount(ctx.damp_kinds) : 1ull;
	if ((uint64_t)nsub * kinds * ctx.ncolours * blocks >= (1ull << 31)) return kNoAllocTooLong;
	e = cudaMemsetAsync(p, ctx.bar_base ? 0xff : 0, sizeof(uint32_t), st);
	if (e == cudaSuccess) e = cudaMemsetAsync(p + 1, 0, sizeof(uint32_t), st);
	if (e != cudaSuccess) return (int)e;
	DevCtx c = ctx;
	c.bar_count = p;
	c.err = reinterpret_cast<int*>(p + 1);
	void* args[] = {&c, &nsub, &dt};
	note_launch(XFEM_FORM_GRID, blocks, (uint32_t)block, 1);
	e = cudaLaunchCooperativeKernel(f, dim3(blocks), dim3(block), args, smem, st);
	if (e != cudaSuccess) return (int)e;
	e = cudaMemcpyAsync(device_error, p + 1, sizeof(int), cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess) e = cudaStreamSynchronize(st);
	return (int)e;
}

}  // namespace xfem
