// bfs_cluster.cu -- the single-source traversal of a small graph in one
// thread-block cluster.
//
// On a graph of a few thousand vertices a step of the whole grid
// (bfs_kernels.cu) is 7 to 10 us of grid barrier, totals and L2 round trips
// around a microsecond of work.  Here one cluster of 1 to 16 CTAs takes the
// whole traversal: the visited, current and next frontier bits of all vertices
// are in every CTA's shared memory, so an edge test is a shared-memory load,
// the barrier is the cluster's own, and frontier bits and totals go from CTA
// to CTA through distributed shared memory.  The steps, their directions and
// all results are those of the grid's kernel (the reference's graph_prepare,
// apps/bfs_simd/bfs.cpp:753-963).
//
// CTA c of C owns the bitmap words c, c + C, c + 2 C, ... (32 vertices each;
// degrees follow the ids in many graphs, so ranges would be uneven).  Per step:
//   bottom-up: the owner of an unvisited vertex scans its in-edges for a
//     frontier source (as phase_pull), then gives its words of the next
//     frontier to every CTA;
//   top-down, small frontier: CTA 0 alone (solo.cuh), as long as it is small;
//   top-down: a CTA expands its own frontier vertices into its own copy of
//     the next frontier; after a barrier the owner of a word ORs the CTAs'
//     copies of it, drops the visited bits and gives it to every CTA.
// The owner writes the levels and adds up the out-degrees of new vertices.
#include <cooperative_groups.h>

#include "bfs_device.cuh"
#include "device_common.cuh"
#include "kernels_api.h"
#include "solo.cuh"

namespace bfsg {

namespace cg = cooperative_groups;

namespace {

constexpr int kClThreads = 1024;
constexpr uint32_t kClWarps = kClThreads / 32;
constexpr uint32_t kClMaxCtas = 16;
constexpr uint32_t kClQueue = 2048;   // per CTA: destinations with in-edges left to scan, vertices to expand
constexpr uint32_t kClWide = 64;      // top-down: vertices of more out-edges are expanded by the whole CTA
constexpr uint32_t kClRounds = 4;     // bottom-up: 32 in-edges of a longer list each, before the whole warp takes it
constexpr uint32_t kClQuick = 4;      // bottom-up: in-edges a lane tests in one round trip before that

struct ClShared {
	uint32_t cnt[3][2];                          // solo lists: vertices, out-edges
	uint32_t count[2][kClMaxCtas];               // by step parity: new vertices of each CTA ...
	unsigned long long deg[2][kClMaxCtas];       // ... and their out-degrees
	unsigned long long solo[4];                  // CTA 0: steps taken, frontier, its out-edges, out-edges inside
	unsigned long long red[5][kClWarps];
	uint32_t nq;                                 // entries of the queue
};

__device__ __forceinline__ unsigned long long block_sum(unsigned long long x, unsigned long long *red) {
	x = warp_sum(x);
	if (lane_id() == 0) red[warp_id()] = x;
	__syncthreads();
	x = warp_sum(lane_id() < kClWarps ? red[lane_id()] : 0ull);
	return x;
}

// A frontier source among the in-edges e, e + stride, ... (eight, below end), or none.
__device__ __forceinline__ uint32_t in_edge_hit(const DevGraph &g, const uint32_t *cur, uint32_t e, uint32_t end,
		uint32_t stride, unsigned long long &tested) {
	uint32_t u[8], hit = 0xFFFFFFFFu;
#pragma unroll
	for (int q = 0; q < 8; ++q) u[q] = e + stride * q < end ? __ldg(g.in_src + e + stride * q) : 0xFFFFFFFFu;
#pragma unroll
	for (int q = 0; q < 8; ++q) {
		if (u[q] == 0xFFFFFFFFu) continue;
		++tested;
		if ((cur[u[q] >> 5] >> (u[q] & 31)) & 1u) hit = u[q];
	}
	return hit;
}

} // namespace

__global__ void __launch_bounds__(kClThreads, 1) k_bfs_cluster(const __grid_constant__ DevGraph g, RunCtx r, StepParams p) {
	extern __shared__ __align__(16) uint32_t dyn[];
	__shared__ ClShared sh;
	cg::cluster_group cl = cg::this_cluster();
	const uint32_t rank = cl.block_rank(), C = cl.num_blocks();
	const uint32_t tid = threadIdx.x, wid = warp_id();
	const unsigned lane = lane_id();
	const uint32_t nw = g.nwords;
	uint32_t *vis = dyn, *cur = vis + nw, *nxt = cur + nw, *queue = nxt + nw, *lists = queue + 3 * kClQueue;
	const uint32_t s = p.source;
	const bool leader = rank == 0 && tid == 0;
	r.vis = nullptr;  // solo.cuh: the visited bits are in shared memory alone
	// statistics of this thread
	unsigned long long td_edges = 0, td_vertices = 0, bu_words = 0, bu_vertices = 0;
	unsigned long long reached = 0, edges = 0;  // leader
	uint32_t dense_steps = 0;

	for (uint32_t w = rank + C * wid; w < nw; w += C * kClWarps) {
		const uint32_t v = w * 32 + lane;
		if (v >= g.n) continue;
		r.level[v] = v == s ? 0 : -1;
		if (r.parent) r.parent[v] = v == s ? s : kUnvisitedWord;
	}
	for (uint32_t w = tid; w < nw; w += kClThreads) vis[w] = cur[w] = w == s / 32 ? 1u << (s & 31) : 0u;
	if (rank == 0)
		for (uint32_t i = tid; i < sizeof(DevStats) / 4; i += kClThreads) ((uint32_t *) r.stats)[i] = 0;
	uint32_t fsize = 1, step = 0, turn = 0;
	unsigned long long dsum = __ldg(g.row_off + s + 1) - __ldg(g.row_off + s), seen = 0;
	bool last_dense = false;
	cl.sync();
	while (fsize) {
		if (leader) {
			reached += fsize;
			edges += dsum;
			if (step < 257) r.stats->t_step[step] = global_timer_ns();
		}
		seen += dsum;
		const bool dense = step > 0 && goes_dense(g, p, fsize, dsum, seen, last_dense);
		if (!dense && fsize <= kSoloCap && dsum <= kSoloCap) {
			// ---- small frontiers: CTA 0, step after step ------------------
			if (rank == 0) {
				if (tid < 6) sh.cnt[tid / 2][tid % 2] = 0;
				__syncthreads();
				for (uint32_t x0 = 0; x0 < nw; x0 += kClThreads) {
					uint32_t bits = x0 + tid < nw ? cur[x0 + tid] : 0u;
					while (__any_sync(kFull, bits)) {
						const bool ok[1] = {bits != 0u};
						uint32_t v[1] = {0}, beg[1] = {0}, deg[1] = {0};
						if (ok[0]) {
							v[0] = (x0 + tid) * 32 + (__ffs(bits) - 1);
							bits &= bits - 1;
							beg[0] = __ldg(g.row_off + v[0]);
							deg[0] = __ldg(g.row_off + v[0] + 1) - beg[0];
						}
						solo_append<1>(solo_list(lists, 0), sh.cnt[0], ok, v, beg, deg);
					}
				}
				__syncthreads();
				uint32_t nv = sh.cnt[0][0], ne = sh.cnt[0][1], done = 0;
				unsigned long long inside = 0;
				for (;;) {
					uint32_t *cn = sh.cnt[(done + 1) % 3];
					if (tid == 0) {
						sh.cnt[(done + 2) % 3][0] = sh.cnt[(done + 2) % 3][1] = 0;
						td_edges += ne;
						td_vertices += nv;
					}
					const SoloList from = solo_list(lists, done & 1), to = solo_list(lists, (done & 1) ^ 1);
					const int32_t nl = (int32_t) (step + done) + 1;
					if (ne <= (uint32_t) kClThreads) solo_expand<1, kClThreads>(g, r, from, to, cn, ne, nl, vis);
					else solo_expand<2, kClThreads>(g, r, from, to, cn, ne, nl, vis);
					__syncthreads();
					++done;
					nv = cn[0];
					ne = cn[1];
					if (nv == 0 || ne > kSoloCap || goes_dense(g, p, nv, ne, seen + inside + ne, false)) break;
					inside += ne;
					if (tid == 0) {
						reached += nv;
						edges += ne;
						if (step + done < 257) r.stats->t_step[step + done] = global_timer_ns();
					}
				}
				for (uint32_t w = tid; w < nw; w += kClThreads) cur[w] = 0;
				__syncthreads();
				const SoloList last = solo_list(lists, done & 1);
				for (uint32_t x = tid; x < nv; x += kClThreads) atomicOr(cur + (last.u[x] >> 5), 1u << (last.u[x] & 31));
				if (tid == 0) {
					sh.solo[0] = done;
					sh.solo[1] = nv;
					sh.solo[2] = ne;
					sh.solo[3] = inside;
				}
			}
			cl.sync();
			if (rank != 0) {
				const uint32_t *rv = cl.map_shared_rank(vis, 0), *rc = cl.map_shared_rank(cur, 0);
				for (uint32_t w = tid; w < nw; w += kClThreads) {
					vis[w] = rv[w];
					cur[w] = rc[w];
				}
			}
			const unsigned long long *rs = cl.map_shared_rank(sh.solo, 0);
			step += (uint32_t) rs[0];
			fsize = (uint32_t) rs[1];
			dsum = rs[2];
			seen += rs[3];
			last_dense = false;
			__syncthreads();
			continue;
		}
		const int32_t nl = (int32_t) step + 1;
		unsigned long long newdeg = 0;
		uint32_t newcount = 0;
		uint32_t *give;  // the array in which every CTA gets the next frontier
		if (dense) {
			// ---- bottom-up --------------------------------------------------
			if (tid == 0) sh.nq = 0;
			for (uint32_t w = rank + C * tid; w < nw; w += C * kClThreads) nxt[w] = 0;
			__syncthreads();
			for (uint32_t w = rank + C * wid; w < nw; w += C * kClWarps) {
				const uint32_t v = w * 32 + lane;
				uint32_t beg = 0, end = 0, u[kClQuick];
				if (v < g.n && !((vis[w] >> lane) & 1u)) {
					beg = __ldg(g.in_off + v);
					end = __ldg(g.in_off + v + 1);
				}
#pragma unroll
				for (uint32_t q = 0; q < kClQuick; ++q) u[q] = beg + q < end ? __ldg(g.in_src + beg + q) : 0xFFFFFFFFu;
				bool found = false;
				uint32_t by = 0;
#pragma unroll
				for (uint32_t q = 0; q < kClQuick; ++q) {
					if (found || u[q] == 0xFFFFFFFFu) continue;
					++bu_words;
					if ((cur[u[q] >> 5] >> (u[q] & 31)) & 1u) {
						found = true;
						by = u[q];
					}
				}
				bu_vertices += beg < end;
				if (found && r.parent) r.parent[v] = by;
				const uint32_t m = __ballot_sync(kFull, found);
				if (lane == 0) nxt[w] = m;
				__syncwarp();
				if (!found && end - beg > kClQuick) {
					const uint32_t at = atomicAdd(&sh.nq, 1u);
					if (at < kClQueue) {
						queue[at] = v;
						queue[kClQueue + at] = beg + kClQuick;
						queue[2 * kClQueue + at] = end;
					} else {  // queue full: finish the scan here
						for (uint32_t e = beg + kClQuick; e < end; ++e) {
							const uint32_t x = __ldg(g.in_src + e);
							++bu_words;
							if ((cur[x >> 5] >> (x & 31)) & 1u) {
								if (r.parent) r.parent[v] = x;
								atomicOr(nxt + w, 1u << lane);
								break;
							}
						}
					}
				}
				__syncwarp();
			}
			__syncthreads();
			// the longer lists: 4 lanes per destination, 8 in-edges per lane and
			// round trip, eight destinations of a warp side by side; what is left
			// of a list after kClRounds of these is the whole warp's (a hub's list
			// would keep its 4 lanes busy long after the step is done)
			const uint32_t nq = min(sh.nq, kClQueue), sub = lane & 3u;
			for (uint32_t x0 = wid * 8; x0 < nq; x0 += kClWarps * 8) {
				const uint32_t x = x0 + lane / 4;
				bool open = x < nq;
				const uint32_t v = open ? queue[x] : 0u, end = open ? queue[2 * kClQueue + x] : 0u;
				uint32_t e = open ? queue[kClQueue + x] : 0u;
				for (uint32_t round = 0; round < kClRounds && __any_sync(kFull, open); ++round) {
					const uint32_t hit = in_edge_hit(g, cur, e + sub, open ? end : 0u, 4, bu_words);
					const uint32_t m = (__ballot_sync(kFull, hit != 0xFFFFFFFFu) >> (lane & 28u)) & 0xFu;
					if (m && sub == (unsigned) __ffs(m) - 1) {
						if (r.parent) r.parent[v] = hit;
						atomicOr(nxt + (v >> 5), 1u << (v & 31));
					}
					e += 32;
					open = open && !m && e < end;
				}
				for (uint32_t om = __ballot_sync(kFull, open && sub == 0); om; om &= om - 1) {
					const int src = __ffs(om) - 1;
					const uint32_t ov = __shfl_sync(kFull, v, src), oend = __shfl_sync(kFull, end, src);
					for (uint32_t oe = __shfl_sync(kFull, e, src); oe < oend; oe += 256) {
						const uint32_t hit = in_edge_hit(g, cur, oe + lane, oend, 32, bu_words);
						const uint32_t m = __ballot_sync(kFull, hit != 0xFFFFFFFFu);
						if (!m) continue;
						if (lane == (unsigned) __ffs(m) - 1) {
							if (r.parent) r.parent[ov] = hit;
							atomicOr(nxt + (ov >> 5), 1u << (ov & 31));
						}
						break;
					}
				}
			}
			__syncthreads();
			give = nxt;
			++dense_steps;
		} else {
			// ---- top-down ---------------------------------------------------
			for (uint32_t w = tid; w < nw; w += kClThreads) nxt[w] = 0;
			if (tid == 0) sh.nq = 0;
			__syncthreads();
			for (uint32_t w = rank + C * wid; w < nw; w += C * kClWarps) {
				const uint32_t bits = cur[w];
				const uint32_t u = w * 32 + lane;
				uint32_t beg = 0, deg = 0;
				if ((bits >> lane) & 1u) {
					beg = __ldg(g.row_off + u);
					deg = __ldg(g.row_off + u + 1) - beg;
					++td_vertices;
					td_edges += deg;
					if (deg > kClWide) {
						const uint32_t at = atomicAdd(&sh.nq, 1u);
						if (at < kClQueue) {
							queue[at] = u;
							deg = 0;
						}
					}
				}
				const uint32_t incl = warp_incl_scan(deg), excl = incl - deg;
				const uint32_t total = __shfl_sync(kFull, incl, 31);
				for (uint32_t f0 = 0; f0 < total; f0 += 128) {
					uint32_t o[4], v[4];
#pragma unroll
					for (int q = 0; q < 4; ++q) {
						const uint32_t f = f0 + 32 * q + lane;
						o[q] = 0;
#pragma unroll
						for (uint32_t st = 16; st; st >>= 1) {
							const uint32_t x = __shfl_sync(kFull, incl, o[q] + st - 1);
							if (x <= f) o[q] += st;
						}
						const uint32_t ob = __shfl_sync(kFull, beg, o[q]), oe = __shfl_sync(kFull, excl, o[q]);
						v[q] = f < total ? __ldg(g.col + ob + (f - oe)) : 0xFFFFFFFFu;
					}
#pragma unroll
					for (int q = 0; q < 4; ++q) {
						if (v[q] == 0xFFFFFFFFu) continue;
						const uint32_t bit = 1u << (v[q] & 31);
						if ((vis[v[q] >> 5] | nxt[v[q] >> 5]) & bit) continue;
						atomicOr(nxt + (v[q] >> 5), bit);
						if (r.parent) r.parent[v[q]] = w * 32 + o[q];
					}
				}
			}
			__syncthreads();
			const uint32_t nq = min(sh.nq, kClQueue);
			for (uint32_t x = 0; x < nq; ++x) {
				const uint32_t u = queue[x];
				const uint32_t beg = __ldg(g.row_off + u), end = __ldg(g.row_off + u + 1);
				for (uint32_t e = beg + tid; e < end; e += 4 * kClThreads) {
					uint32_t v[4];
#pragma unroll
					for (int q = 0; q < 4; ++q) v[q] = e + q * kClThreads < end ? __ldg(g.col + e + q * kClThreads) : 0xFFFFFFFFu;
#pragma unroll
					for (int q = 0; q < 4; ++q) {
						if (v[q] == 0xFFFFFFFFu) continue;
						const uint32_t bit = 1u << (v[q] & 31);
						if ((vis[v[q] >> 5] | nxt[v[q] >> 5]) & bit) continue;
						atomicOr(nxt + (v[q] >> 5), bit);
						if (r.parent) r.parent[v[q]] = u;
					}
				}
			}
			cl.sync();
			give = cur;  // nobody reads the old frontier any more
		}
		// ---- the owned words of the next frontier: to every CTA; levels; totals
		for (uint32_t w = rank + C * wid; w < nw; w += C * kClWarps) {
			const uint32_t bits = dense ? nxt[w]
					: __reduce_or_sync(kFull, lane < C ? cl.map_shared_rank(nxt, lane)[w] : 0u) & ~vis[w];
			if (lane < C && (lane != rank || !dense)) cl.map_shared_rank(give, lane)[w] = bits;
			if ((bits >> lane) & 1u) {
				const uint32_t v = w * 32 + lane;
				newdeg += __ldg(g.row_off + v + 1) - __ldg(g.row_off + v);
				++newcount;
				r.level[v] = nl;
			}
		}
		// the two sums in one block reduction: counts are at most 2^17
		const unsigned long long both = block_sum(newdeg | ((unsigned long long) newcount << 40), sh.red[0]);
		if (tid < C) {
			cl.map_shared_rank(&sh.count[0][0], tid)[turn * kClMaxCtas + rank] = (uint32_t) (both >> 40);
			cl.map_shared_rank(&sh.deg[0][0], tid)[turn * kClMaxCtas + rank] = both & ((1ull << 40) - 1);
		}
		cl.sync();
		fsize = 0;
		dsum = 0;
		for (uint32_t c = 0; c < C; ++c) {
			fsize += sh.count[turn][c];
			dsum += sh.deg[turn][c];
		}
		turn ^= 1u;
		if (dense) {
			uint32_t *t = cur;
			cur = nxt;
			nxt = t;
		}
		for (uint32_t w = tid; w < nw; w += kClThreads) vis[w] |= cur[w];
		__syncthreads();
		if (leader && step < 256) r.stats->trace[step] = dense ? 1 : 0;
		++step;
		last_dense = dense;
	}
	// statistics, CTA by CTA
	const unsigned long long mine[4] = {td_edges, td_vertices, bu_words, bu_vertices};
	unsigned long long *const out[4] = {&r.stats->td_edges, &r.stats->td_vertices, &r.stats->bu_words, &r.stats->bu_vertices};
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		const unsigned long long t = block_sum(mine[i], sh.red[i + 1]);
		if (tid == 0 && t) atomicAdd(out[i], t);
	}
	if (leader) {
		if (step < 257) r.stats->t_step[step] = global_timer_ns();
		r.stats->reached = reached;
		r.stats->edges_traversed = edges;
		r.stats->dense_steps = dense_steps;
		r.stats->num_steps = step;
		r.stats->status = 0;
	}
	cl.sync();  // nobody's shared memory goes before the others have read it
}

namespace {

size_t cluster_smem(const DevGraph &g) { return sizeof(uint32_t) * ((size_t) 3 * g.nwords + 3 * kClQueue + kSoloWords); }

int cluster_config(const DevGraph &g, int ctas, cudaStream_t st, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr) {
	attr->id = cudaLaunchAttributeClusterDimension;
	attr->val.clusterDim.x = (unsigned) ctas;
	attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
	*cfg = cudaLaunchConfig_t{};
	cfg->gridDim = dim3((unsigned) ctas);
	cfg->blockDim = dim3(kClThreads);
	cfg->dynamicSmemBytes = cluster_smem(g);
	cfg->stream = st;
	cfg->attrs = attr;
	cfg->numAttrs = 1;
	return BFS_OK;
}

} // namespace

int cluster_ctas(const DevGraph &g) {
	if (g.n > kClusterMaxVertices || g.m > kClusterMaxEdges) return 0;
	if (g.n > kClusterDenseVertices && (uint64_t) g.m > (uint64_t) kClusterSparseDegree * g.n) return 0;
	int ctas = 1;
	while (ctas < (int) kClMaxCtas && (uint32_t) ctas * kClusterVerticesPerCta < g.n) ctas *= 2;
	const size_t most = sizeof(uint32_t) * ((size_t) 3 * ((kClusterMaxVertices + 31) / 32) + 3 * kClQueue + kSoloWords);
	if (cudaFuncSetAttribute(k_bfs_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) most) != cudaSuccess ||
			cudaFuncSetAttribute(k_bfs_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
		cudaGetLastError();
		return 0;
	}
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute attr;
	cluster_config(g, ctas, nullptr, &cfg, &attr);
	int clusters = 0;
	if (cudaOccupancyMaxActiveClusters(&clusters, k_bfs_cluster, &cfg) != cudaSuccess || clusters < 1) {
		cudaGetLastError();
		return 0;
	}
	return ctas;
}

int launch_cluster(const DevGraph &g, const RunCtx &r, const StepParams &p, int ctas, cudaStream_t st) {
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute attr;
	cluster_config(g, ctas, st, &cfg, &attr);
	return cudaLaunchKernelEx(&cfg, k_bfs_cluster, g, r, p) == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

} // namespace bfsg
