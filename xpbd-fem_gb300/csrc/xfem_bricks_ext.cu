// The tet kernel with damping and volume sweeps on the bricks (sm_103a): handles
// whose bodies damp after the solves or run volume passes, all of them with the
// plain solve, on meshes whose clusters are all whole cubes. Where the plain solve would run k_bricks (xfem_kernels.cu)
// such a handle ran the grid form: a barrier over 152 blocks per pass, and every
// vertex through L2. Here each block keeps its brick's own vertices in shared
// memory, interior chunks start at once, and a boundary chunk waits for the
// neighbouring bricks: for all of them, because with damping passes that are
// skipped when nothing is damped at a tick, which brick touched a vertex last
// changes from pass to pass. Colours, clusters and arithmetic are k_persistent's;
// the results are bit-identical.
//
// Bound by the chain of a pass: a boundary warp's 7,600 cycles for a solve and
// 8,800 for a damping pass (the brick has 2.6 chunks of a colour, on as many
// warps), and 2,000 to 4,500 until the neighbours' pass counts are there.
// Measured, a frame of 20 substeps with the interactive damping settings, grid
// form before: 608,256 tets 1,872 -> 1,396 us, 3,145,728 tets (two bricks per SM)
// 3,808 -> 2,510.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "xfem_chunk.cuh"
#include "xfem_device.cuh"
#include "xfem_internal.h"

namespace xfem {

namespace {

// Element sweeps of a substep, in their order.
enum class Sweep { kSolve, kVolume, kRayleigh, kPbd };

__device__ __forceinline__ Sweep sweep_of(const DevCtx& C, uint32_t kind) {
	return kind == 0 ? Sweep::kSolve : kind <= C.nvol ? Sweep::kVolume : damp_kind(C, kind) == 0 ? Sweep::kRayleigh : Sweep::kPbd;
}

// A pass of any sweep over a resident chunk of whole cubes, for handles whose
// bodies all have the plain solve: the solves, a volume sweep (k: its 1-based
// number) or a damping sweep. The same steps as run_chunk, vol_chunk and
// damp_chunk, but one load of the eight vertices and one write-back for all of
// them. With those three inlined or called side by side the kernel kept its
// registers on the stack (1,040 bytes, 160 of them spilled) and a damped frame of
// 608,256 tets took 1,773 us; so, with no stack, 1,515 then.
template <class VS, class BP>
__device__ __forceinline__ void sweep_cube(const DevCtx& C, const VS& vs, const BP& bps, Stage& st, const BrickLane& bl, uint32_t chunk, int next,
                                           uint32_t lane, Sweep sweep, uint32_t k, bool first, bool finish, float dt,
                                           float inv_dt, float inv_dt2, uint32_t tick) {
	const uint32_t trow = chunk * 6u;
	const float4* rec = reinterpret_cast<const float4*>(st.buf);
	const uint32_t hdr = bl.hdr;
	const uint32_t* vid = bl.vw;
	const bool live = (hdr & 15u) != 0, solve = sweep == Sweep::kSolve;
	const uint32_t mask = solve ? (hdr >> 8) & 0xffu : 0u;
	float4 O[8], D[8];  // a damping sweep's X and V
	uint32_t last = 0;  // the vertices that this pass finishes, with damping sweeps
	uint32_t some = 0;  // bit t: tet t has work
	if (live) {
#pragma unroll
		for (int s = 0; s < 8; s++) vs.ld(C, vid[s], O[s], D[s]);
		const Mat mat = bps.mat(C, hdr >> 16);
		DampBody d = {false, false, 0.0f, 0.0f, 0u, 0u};
		float ar = 0.0f;  // PBD: the area of the tet that is next
		if (solve || sweep == Sweep::kVolume) {
			// the body's last volume sweep finishes, or, without any, its solve
			if (finish && mat.nvol == k) last = __ldg(C.blastmask + (size_t)chunk * kLanes + lane);
			if (solve || mat.nvol >= k) some = 63u;
		} else {
			d = damp_of(C.bodies[hdr >> 16], tick, sweep == Sweep::kRayleigh ? 0 : 1);
			if (d.on) {
				if (sweep == Sweep::kPbd) ar = __ldg(C.btarea + (size_t)trow * kLanes + lane);
#pragma unroll
				for (uint32_t t = 0; t < 6; t++) {
					const uint32_t f = d.amort ? __ldg(C.btflat + (size_t)(trow + t) * kLanes + lane) : 0u;
					if (!d.amort || (f >= d.lo && f < d.hi)) some |= 1u << t;
				}
			}
		}
#pragma unroll
		for (int s = 0; s < 8; s++)
			if (mask & (1u << s)) bps.advance(C, vs.id(vid[s]), O[s], D[s], first, dt, inv_dt);
		if (solve) {
			solve_cube<false>(
			    mat, rec + lane, inv_dt, inv_dt2, O, D, [](int, const float4*) {}, [](int, const float2&) {});
		} else if (sweep == Sweep::kVolume) {
			if (some)
				turn_cube(O, D, [&](int t, const float4* Ot, float4* Dt) {
					volume_tet(mat, cluster_rec(rec + lane, t), inv_dt2, Ot, Dt);
				});
		} else if (sweep == Sweep::kRayleigh) {
			if (some)
				turn_cube(O, D, [&](int t, const float4* Xt, float4* Vt) {
					if (some >> t & 1u) rayleigh_tet<false>(mat, cluster_rec(rec + lane, t), Xt, Vt, inv_dt, d.rayleigh);
				});
		} else if (some) {
			turn_cube(O, D, [&](int t, const float4* Xt, float4* Vt) {
				const float a = ar;
				if (t < 5) ar = __ldg(C.btarea + (size_t)(trow + t + 1) * kLanes + lane);
				if (some >> t & 1u) pbd_tet(Xt, Vt, fminf(1.0f, d.pbd / a));
			});
		}
	}
	if (next >= 0) brick_issue(C, st, (uint32_t)next, lane);  // buffer consumed: prefetch
	if (some) {
#pragma unroll
		for (int s = 0; s < 8; s++) {
			if (last & (1u << s)) bps.finalize(C, vs.id(vid[s]), O[s], D[s], inv_dt);
			vs.st(C, vid[s], O[s], D[s], ((mask | last) & (1u << s)) != 0u);
		}
	}
}

// Two bricks of 192 threads per SM, or one of 256.
template <bool ONE, bool PAIR>
__global__ void __launch_bounds__(PAIR ? 192 : 256, PAIR ? 2 : 1) k_bricks_ext(const __grid_constant__ DevCtx C, uint32_t nsub, float dt) {
	extern __shared__ __align__(128) uint8_t smem[];
	__shared__ uint32_t s_bcb[65], s_bwait[64];
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	const uint32_t b = blockIdx.x, ncol = C.ncolours;
	const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
	const uint32_t tick0 = __ldcg(C.tick);  // read before this brick publishes; block 0 advances it at the end
	const bool dmode = C.damp_kinds != 0u;
	const uint32_t P = pass_kinds(C) * ncol;
	Stage st = brick_stage_init(lane);
	float4* sv = reinterpret_cast<float4*>(smem + (size_t)wpb * kBrickChunkBytes);
	uint32_t* spid = reinterpret_cast<uint32_t*>(sv + 2 * (size_t)C.bpriv_max);
	const BrickVerts<!PAIR> vs = {sv, spid, C.bpriv_max};
	const auto bps = body_params<ONE>(C);
	for (uint32_t i = threadIdx.x; i <= ncol; i += blockDim.x) {
		s_bcb[i] = __ldg(C.bchunk_begin + (size_t)b * ncol + i);
		if (i < ncol) s_bwait[i] = __ldg(C.bchunk_wait_end + (size_t)b * ncol + i);
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
	run_isolated(C, GlobalVerts{}, gtid, nthreads, nsub, dt, inv_dt, true);
	const uint32_t nb0 = __ldg(C.bnb_begin + b), nb1 = __ldg(C.bnb_begin + b + 1);
	uint32_t epoch = 0;
	bool ok = true;
	// the warp's next chunk after `ch`, pass q of substep s (-1: none)
	auto next_of = [&](uint32_t ch, uint32_t q, uint32_t s) {
		if (ch + wpb < s_bcb[q % ncol + 1]) return (int)(ch + wpb);
		for (uint32_t k = 0; k < P; k++) {
			if (++q == P) q = 0, s++;
			if (s >= nsub) return -1;
			if (q >= ncol && !pass_runs(C, q, tick0 + s)) continue;
			const uint32_t f = s_bcb[q % ncol] + wib;
			if (f < s_bcb[q % ncol + 1]) return (int)f;
		}
		return -1;
	};
	for (uint32_t s = 0; s < nsub && ok; s++) {
		for (uint32_t q = 0; q < P && ok; q++) {
			const uint32_t kind = q / ncol, c = q - kind * ncol;
			if (kind > 0 && !pass_runs(C, q, tick0 + s)) continue;  // the same in every brick
			const uint32_t wend = s_bwait[c];
			bool bad = false, waited = false;
			for (uint32_t ch = s_bcb[c] + wib; ch < s_bcb[c + 1] && !bad; ch += wpb) {
				if (!brick_acquire(C, st, ch, lane)) {
					bad = true;
					break;
				}
				const int next = next_of(ch, q, s);
				BrickLane bl;
				if (!PAIR) bl = brick_lane(st, lane);
				if (ch < wend && !waited) {
					bad = __any_sync(0xffffffffu, !brick_wait(C, C.bnb, nb0, nb1, epoch, lane, 32u));
					__syncwarp();  // orders every lane's loads after the lanes' acquires
					waited = true;
					if (bad) break;
				}
				if (PAIR) bl = brick_lane(st, lane);
				sweep_cube(C, vs, bps, st, bl, ch, next, lane, sweep_of(C, kind), kind, dmode || s == 0, dmode, dt, inv_dt, inv_dt2,
				           tick0 + s);
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
	// with damping sweeps the state is canonical; else the last substep is
	// finalized here, each brick its own vertices and its share of the others
	for (uint32_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
		const uint32_t v = spid[i - pb];
		float4 O = sv[i - pb], D = sv[C.bpriv_max + (i - pb)];
		if (!dmode) bps.finalize(C, v, O, D, inv_dt);
		st_vertex(C.vert + 2 * (size_t)v, O, D);
	}
	if (!dmode) {
		const uint32_t fb = __ldg(C.bfin_begin + b), fe = __ldg(C.bfin_begin + b + 1);
		for (uint32_t i = fb + threadIdx.x; i < fe; i += blockDim.x) {
			const uint32_t v = __ldg(C.bfin_vid + i);
			float4 O, D;
			ld_vertex(C.vert + 2 * (size_t)v, O, D);
			bps.finalize(C, v, O, D, inv_dt);
			st_vertex(C.vert + 2 * (size_t)v, O, D);
		}
	}
	// the tick moves on once every brick, also of other bodies, has read it: each
	// did before it published its first pass
	if (b == 0) {
		ok = !__syncthreads_or(brick_wait<true>(C, nullptr, 0, C.nbricks, 1u, threadIdx.x, blockDim.x) ? 0 : 1);
		if (ok && threadIdx.x == 0) *C.tick = tick0 + nsub;
	}
}

__global__ void k_brick_sweeps(DevCtx C, const uint32_t* __restrict__ src, uint32_t n, uint32_t* __restrict__ lastmask,
                               uint32_t* __restrict__ flat, float* __restrict__ area) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint32_t from = src[i], chunk = i / kLanes, lane = i % kLanes;
	const bool on = from != kNoLane;
	const uint32_t trow = on ? C.chunks[from / kLanes].trow : 0u;
	lastmask[i] = on ? C.lastmask[from] : 0u;
	for (uint32_t t = 0; t < 6; t++) {
		const size_t to = ((size_t)chunk * 6 + t) * kLanes + lane, at = ((size_t)trow + t) * kLanes + from % kLanes;
		flat[to] = on ? C.tflat[at] : 0u;
		area[to] = on ? C.tarea[at] : 0.0f;
	}
}

const void* brick_ext_fn(bool one, bool pair) {
	if (pair) return one ? (const void*)k_bricks_ext<true, true> : (const void*)k_bricks_ext<false, true>;
	return one ? (const void*)k_bricks_ext<true, false> : (const void*)k_bricks_ext<false, false>;
}

}  // namespace

int launch_brick_sweeps(const DevCtx& ctx, const uint32_t* src, uint32_t n, uint32_t* lastmask, uint32_t* flat, float* area,
                        void* stream) {
	if (!n) return 0;
	k_brick_sweeps<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(ctx, src, n, lastmask, flat, area);
	return (int)cudaGetLastError();
}

// Whether the bricks run at once at this block size. Two bricks per SM have blocks
// of 192 threads at most: 168 registers a thread.
int brick_ext_fits(const DevCtx& C, int block, bool* fits) {
	*fits = false;
	int dev = 0, sms = 0, per_sm = 0, optin = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
	if (e != cudaSuccess) return (int)e;
	const bool pair = C.nbricks > (uint32_t)sms;
	if (!C.nbricks || (block != 128 && block != 192 && block != 224 && block != 256) || (pair && block > 192)) return 0;
	const void* f = brick_ext_fn(C.nbodies == 1, pair);
	cudaFuncAttributes fa{};
	if ((e = cudaFuncGetAttributes(&fa, f)) != cudaSuccess) return (int)e;
	const size_t smem = brick_smem_bytes(block, C.bpriv_max);
	if (smem + fa.sharedSizeBytes > (size_t)optin) return 0;
	e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, block, smem);
	if (e == cudaSuccess) *fits = (uint64_t)per_sm * (uint64_t)sms >= C.nbricks;
	return (int)e;
}

int launch_bricks_ext(const DevCtx& ctx, int block, uint32_t nsub, float dt, void* stream) {
	cudaStream_t st = (cudaStream_t)stream;
	int dev = 0, sms = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (e != cudaSuccess) return (int)e;
	const void* f = brick_ext_fn(ctx.nbodies == 1, ctx.nbricks > (uint32_t)sms);
	const size_t smem = brick_smem_bytes(block, ctx.bpriv_max);
	// pass counters start at 0; one launch counts at most 2^30 passes
	const uint32_t kinds = 1u + ctx.nvol + (uint32_t)__builtin_popcount(ctx.damp_kinds);
	const uint32_t per = std::max(1u, (1u << 30) / std::max(1u, kinds * ctx.ncolours));
	for (uint32_t done = 0; done < nsub;) {
		uint32_t n = std::min(per, nsub - done);
		e = cudaMemsetAsync(ctx.bflag, 0, sizeof(uint32_t) * kBrickFlagStride * ctx.nbricks, st);
		if (e != cudaSuccess) return (int)e;
		DevCtx c = ctx;
		float dtv = dt;
		void* args[] = {&c, &n, &dtv};
		note_launch(XFEM_FORM_BRICKS_EXT, ctx.nbricks, (uint32_t)block, 1);
		e = cudaLaunchCooperativeKernel(f, dim3(ctx.nbricks), dim3(block), args, smem, st);
		if (e != cudaSuccess) return (int)e;
		done += n;
	}
	return 0;
}

}  // namespace xfem
