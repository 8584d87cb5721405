// The one-cluster form of the persistent tet kernel (sm_103a), for small
// handles (sync_mode 1 and the adjoint's recording forward).
//
// A colour pass of a small body is one chunk's chain of gathers and solves per
// warp. In the grid form the pass also pays a barrier over 152 blocks (1.4 us),
// the vertices' way to L2 and back (0.7 us each) and the copy of the chunk's
// records. Here the whole grid is one thread-block cluster of at most 16
// blocks: every vertex stays in its distributed shared memory for the launch,
// a pass ends at the hardware cluster barrier, and each warp has its chunks'
// records in several buffers, all of them resident when they fit.
//
// Block r takes the r-th run of each colour's chunks, one per warp, and holds
// the r-th run of the vertices; both lie along the Morton curve, so most of a
// chunk's vertices are its own block's. The colours, chunks and arithmetic are
// k_persistent's: the results are bit-identical.
//
// What is left of a pass is the chain of a warp's instructions (gather, six to
// eight dependent solves, write-back). Measured (one frame, GB300; before: the
// fastest other form): 192 tets, 1 block, 656 -> 468 us (2.9 us per pass);
// 98,304 tets, 16 blocks of 4 chunk warps, 1,172 -> 1,033 us; 78,336 tets in
// clusters of every shape (20 colours) 2,427 -> 2,008 us; 6,144 damped tets, a
// launch per substep, 967 -> 702 us for ten; the recording forward of 12,288
// tets x 200 substeps 9.7 -> 6.1 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "xfem_chunk.cuh"
#include "xfem_device.cuh"
#include "xfem_internal.h"

namespace xfem {

namespace {

constexpr uint32_t kClusterBufs = 8;     // chunk buffers of a warp, at most
constexpr uint32_t kClusterColours = 24;  // colours whose chunk descriptors sit in shared memory

// A warp's shared memory: its chunk buffers, then the vertex slots.
XFEM_HD uint32_t cluster_warp_bytes(uint32_t vs_off, uint32_t warp_smem, uint32_t bufs) {
	return bufs * vs_off + (warp_smem - vs_off);
}

// ONE: a single body, its parameters in registers.
template <bool TAPE, int LEVEL, bool ONE>
__global__ void __launch_bounds__(256) k_cluster(DevCtx C, ClusterPlan plan, uint32_t nsub, float dt) {
	extern __shared__ __align__(128) uint8_t smem[];
	__shared__ uint64_t s_mbar[8][kClusterBufs];
	__shared__ int s_ch[8][kClusterColours];
	__shared__ uint4 s_meta[8][kClusterColours];
	const float inv_dt = 1.0f / dt, inv_dt2 = 1.0f / (dt * dt);
	const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
	const uint32_t G = gridDim.x, r = blockIdx.x;
	const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
	constexpr bool EXT = LEVEL != 0;
	const bool dmode = EXT && C.damp_kinds != 0u;
	const uint32_t ncol = C.ncolours, P = (EXT ? pass_kinds(C) : 1u) * ncol, nbuf = plan.bufs;
	const uint32_t tick0 = __ldcg(C.tick);  // read before the first barrier; block 0 advances it at the end
	const auto bps = body_params<ONE>(C);

	// the block's vertices
	const uint32_t wbytes = cluster_warp_bytes(C.vs_off, C.warp_smem, nbuf);
	float4* sv = reinterpret_cast<float4*>(smem + (size_t)plan.warps * wbytes);
	const uint32_t per = cluster_verts(C.nverts, G);
	const ClusterVerts vs(smem_u32(sv), per);
	const uint32_t v0 = min(r * per, C.nverts), v1 = min(v0 + per, C.nverts);
	for (uint32_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
		float4 O, D;
		ld_vertex(C.vert + 2 * (size_t)v, O, D);
		sv[v - v0] = O;
		sv[per + (v - v0)] = D;
	}

	// the warp's chunk of each colour (-1: none) and its descriptor
	auto find_chunk = [&](uint32_t c) {
		const uint32_t cb = __ldg(C.colour_chunk_begin + c), n = __ldg(C.colour_chunk_begin + c + 1) - cb;
		const uint32_t i = n * r / G + wib;
		return i < n * (r + 1u) / G ? (int)(cb + i) : -1;
	};
	auto load_meta = [&](int ch) { return __ldg(reinterpret_cast<const uint4*>(C.chunks) + ch); };
	for (uint32_t c = lane; c < min(ncol, kClusterColours); c += 32u) {
		const int ch = find_chunk(c);
		s_ch[wib][c] = ch;
		if (ch >= 0) s_meta[wib][c] = load_meta(ch);
	}
	uint8_t* wbuf = smem + (size_t)wib * wbytes;
	if (wib < plan.warps && lane < nbuf) mbar_init(&s_mbar[wib][lane]);
	__syncwarp();
	auto chunk_of = [&](uint32_t c) { return c < kClusterColours ? s_ch[wib][c] : find_chunk(c); };
	auto meta_of = [&](uint32_t c, int ch) { return c < kClusterColours ? s_meta[wib][c] : load_meta(ch); };

	// The records: resident (buffer c holds colour c's chunk) or a ring, where
	// the copy of the warp's chunk nbuf - 1 passes ahead is issued at the start
	// of a pass, into the buffer that the pass before it has read.
	const bool resident = nbuf >= ncol;
	uint32_t ps = 0, pq = 0, issued = 0, used = 0;  // the next pass to issue for; copies issued and consumed
	bool ok = true;
	auto issue = [&](uint32_t b, const uint4& m) {
		__syncwarp();
		if (lane == 0) bulk_copy_g2s(wbuf + (size_t)b * C.vs_off, C.cblk + m.x, m.y, &s_mbar[wib][b]);
	};
	auto issue_next = [&]() {
		for (; ps < nsub; ps++, pq = 0) {
			for (; pq < P; pq++) {
				const uint32_t c = pq % ncol;
				const int ch = chunk_of(c);
				if (ch < 0 || (EXT && pq >= ncol && !pass_runs(C, pq, tick0 + ps))) continue;
				issue(issued % nbuf, meta_of(c, ch));
				issued++;
				pq++;
				return;
			}
		}
	};
	const bool works = wib < plan.warps;
	if (works) {
		if (resident) {
			for (uint32_t c = 0; c < ncol; c++)
				if (const int ch = chunk_of(c); ch >= 0) issue(c, meta_of(c, ch));
		} else {
			for (uint32_t k = 0; k + 1 < nbuf; k++) issue_next();
		}
	}
	cluster_barrier();
	run_isolated<TAPE>(C, vs, gtid, nthreads, nsub, dt, inv_dt, dmode);

	for (uint32_t s = 0; s < nsub; s++) {
		for (uint32_t q = 0; q < P; q++) {
			const uint32_t kind = q / ncol, c = q - kind * ncol;
			if (EXT && kind > 0 && !pass_runs(C, q, tick0 + s)) continue;  // the same in every block
			const int ch = works ? chunk_of(c) : -1;
			// a copy that failed ends the warp's work, but not its barriers:
			// every thread of the cluster reaches each of them
			if (ch >= 0 && ok) {
				uint32_t b = c, parity = 0;
				if (!resident) {
					issue_next();
					b = used % nbuf;
					parity = used / nbuf & 1u;
					used++;
				}
				ok = mbar_wait(C, &s_mbar[wib][b], parity);
				Stage st = {wbuf + (size_t)b * C.vs_off, reinterpret_cast<float4*>(wbuf + (size_t)nbuf * C.vs_off), nullptr, 0u,
				            -1, meta_of(c, ch)};
				if (!ok)
					;
				else if (!EXT || kind == 0)
					run_chunk<false, TAPE, EXT, LEVEL == 2>(C, vs, bps, st, (uint32_t)ch, -1, lane, dmode || s == 0, dt,
					                                                    inv_dt, inv_dt2, s, dmode);
				else if (kind <= C.nvol)
					run_vol_chunk(C, vs, st, (uint32_t)ch, -1, lane, inv_dt, inv_dt2, kind, dmode);
				else
					run_damp_chunk(C, vs, st, -1, lane, damp_kind(C, kind), inv_dt, tick0 + s);
			}
			cluster_barrier();
		}
	}
	if (works && !ok) {  // leave no copy in flight
		for (uint32_t k = used; k < issued; k++) mbar_wait(C, &s_mbar[wib][k % nbuf], k / nbuf & 1u);
		for (uint32_t c = 0; resident && c < ncol; c++)
			if (chunk_of(c) >= 0) mbar_wait(C, &s_mbar[wib][c], 0u);
	}
	if (dmode) {
		for (uint32_t v = v0 + threadIdx.x; v < v1; v += blockDim.x)
			st_vertex(C.vert + 2 * (size_t)v, sv[v - v0], sv[per + (v - v0)]);
	} else {
		run_finalize<TAPE>(C, vs, v0 + threadIdx.x, v1, blockDim.x, inv_dt, nsub);
	}
	if (gtid == 0) *C.tick = tick0 + nsub;
}

const void* cluster_fn(bool tape, int ext, bool one) {
	if (tape) return one ? (const void*)k_cluster<true, 0, true> : (const void*)k_cluster<true, 0, false>;
	if (ext == 2) return one ? (const void*)k_cluster<false, 2, true> : (const void*)k_cluster<false, 2, false>;
	if (ext == 1) return one ? (const void*)k_cluster<false, 1, true> : (const void*)k_cluster<false, 1, false>;
	return one ? (const void*)k_cluster<false, 0, true> : (const void*)k_cluster<false, 0, false>;
}

size_t cluster_smem(const DevCtx& C, const ClusterPlan& p) {
	return (size_t)p.warps * cluster_warp_bytes(C.vs_off, C.warp_smem, p.bufs) + 32u * (size_t)cluster_verts(C.nverts, p.blocks);
}

void cluster_config(const DevCtx& C, const ClusterPlan& p, int block, cudaLaunchAttribute* at, cudaLaunchConfig_t* lc) {
	at->id = cudaLaunchAttributeClusterDimension;
	at->val.clusterDim.x = p.blocks;
	at->val.clusterDim.y = at->val.clusterDim.z = 1;
	lc->gridDim = dim3(p.blocks);
	lc->blockDim = dim3(block);
	lc->dynamicSmemBytes = cluster_smem(C, p);
	lc->attrs = at;
	lc->numAttrs = 1;
}

}  // namespace

// The rule: every chunk of the largest colour its own warp (a second round of
// chunks per pass costs what the barrier saves: 98,304 tets at 64 threads a
// block, which fall to the grid form, take 1,572 us against 1,064), at least
// two chunk buffers a warp (with one, the next chunk's copy is waited for:
// 192 tets 753 us against 494), every vertex in shared memory. Of the cluster
// sizes that allow it: the smallest whose blocks hold all their records with
// at most one chunk warp per scheduler, else the largest.
int cluster_plan(const DevCtx& C, uint32_t max_colour_chunks, int block, bool tape, int ext, ClusterPlan* plan) {
	*plan = ClusterPlan();
	if (block > 256 || block % 32 || C.nverts == 0 || C.ncolours == 0) return 0;
	int dev = 0, optin = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
	const void* f = cluster_fn(tape, ext, C.nbodies == 1);
	cudaFuncAttributes fa{};
	if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f);
	if (e != cudaSuccess) return (int)e;
	ClusterPlan best;
	for (uint32_t G = 1; G <= 16; G *= 2) {
		ClusterPlan p;
		p.blocks = G;
		p.warps = (max_colour_chunks + G - 1) / G;
		if (p.warps > (uint32_t)block / 32u) continue;
		// the records of every colour, or two buffers
		p.bufs = C.ncolours <= kClusterBufs ? C.ncolours : 2u;
		if (cluster_smem(C, p) + fa.sharedSizeBytes > (size_t)optin) p.bufs = std::min(2u, C.ncolours);
		if (cluster_smem(C, p) + fa.sharedSizeBytes > (size_t)optin) continue;
		best = p;
		if (p.warps <= 4 && p.bufs >= C.ncolours) break;
		if (p.warps <= 1) break;
	}
	if (!best.blocks) return 0;
	cudaLaunchAttribute at{};
	cudaLaunchConfig_t lc{};
	cluster_config(C, best, block, &at, &lc);
	// the limit is the kernel's on this device: only ever raised, to what the device allows
	e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
	int n = 0;
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, f, &lc);
	if (e != cudaSuccess) return (int)e;
	if (n > 0) *plan = best;
	return 0;
}

// Not a cooperative launch: the blocks of a cluster are always resident together.
int launch_cluster(const DevCtx& ctx, const ClusterPlan& plan, int block, bool tape, int ext, uint32_t nsub, float dt,
                   void* stream) {
	cudaLaunchAttribute at{};
	cudaLaunchConfig_t lc{};
	cluster_config(ctx, plan, block, &at, &lc);
	lc.stream = (cudaStream_t)stream;
	DevCtx c = ctx;
	ClusterPlan p = plan;
	void* args[] = {&c, &p, &nsub, &dt};
	note_launch(XFEM_FORM_CLUSTER, plan.blocks, (uint32_t)block, 1);
	return (int)cudaLaunchKernelExC(&lc, cluster_fn(tape, ext, ctx.nbodies == 1), args);
}

}  // namespace xfem
