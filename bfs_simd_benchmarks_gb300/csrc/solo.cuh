// solo.cuh -- top-down BFS steps by one CTA, the frontier in shared memory.
//
// Used while a frontier is small by the traversal of the whole grid
// (bfs_kernels.cu) and by the one-cluster traversal of small graphs
// (bfs_cluster.cu).  A step of up to 512 edges is two round trips (edge; claim
// and row offsets) and one block barrier: 1.05 us against 6.9 us of the grid
// (1.9 us with the claim as a compare-and-swap on the level in L2, as graphs
// too large for the visited bits in shared memory take it).  A 301 x 287
// street grid of 395 levels: 2.78 -> 0.79 ms.
#pragma once

#include <cstdint>

#include "bfs_device.cuh"
#include "device_common.cuh"

namespace bfsg {

// The direction of the step that expands this frontier (apps/bfs_simd/bfs.cpp:
// 829-834, or Beamer's rule); `seen` includes the frontier's own out-edges.
__device__ __forceinline__ bool goes_dense(const DevGraph &g, const StepParams &p, uint32_t fsize,
		unsigned long long dsum, unsigned long long seen, bool last_dense) {
	if (p.switch_rule == 0) {
		const unsigned long long thr = last_dense ? p.to_sparse_threshold : p.to_dense_threshold;
		return (unsigned long long) fsize + dsum > thr;
	}
	const unsigned long long unseen = g.m > seen ? g.m - seen : 0ull;
	return last_dense ? (unsigned long long) fsize * p.beta >= g.n : dsum * p.alpha > unseen;
}

// Largest frontier: at 2048 edges a step takes about as long as half a step of
// the grid, and the five words per edge of two lists still fit the shared
// memory that the grid's own top-down step uses.
constexpr uint32_t kSoloCap = 2048;
constexpr uint32_t kSoloWords = 5 * kSoloCap;  // dynamic shared memory of its lists ...
constexpr uint32_t kSoloVisWords = 8192;       // ... and of the visited bits of graphs of at most 2^18 vertices
static_assert(kSoloCap <= 0x10000, "owners are 16-bit");

// One of the two frontier lists: vertex u[x] owns the out-edge slots off ..
// off + deg - 1 of its list, fb[x] = (first edge) - off, owner[slot] = x.
struct SoloList {
	uint32_t *u, *fb;
	uint16_t *owner;
};
__device__ __forceinline__ SoloList solo_list(uint32_t *smem, uint32_t which) {
	uint32_t *b = smem + (size_t) which * (kSoloWords / 2);
	return {b, b + kSoloCap, (uint16_t *) (b + 2 * kSoloCap)};
}

// Appends the lanes' vertices v[q] (ok[q]; out-edges beg[q], deg[q]) to `l`;
// cnt[0], cnt[1]: its vertices and out-edges.  All 32 lanes call it.  Slots
// past kSoloCap are not filled: a list with more edges is never expanded here.
template <int Q>
__device__ __forceinline__ void solo_append(const SoloList &l, uint32_t *cnt, const bool (&ok)[Q], const uint32_t (&v)[Q],
		const uint32_t (&beg)[Q], const uint32_t (&deg)[Q]) {
	const unsigned lane = lane_id();
	uint32_t c = 0, d = 0;
#pragma unroll
	for (int q = 0; q < Q; ++q) {
		c += ok[q];
		d += ok[q] ? deg[q] : 0u;
	}
	if (!__ballot_sync(kFull, c)) return;
	const uint32_t ci = warp_incl_scan(c), di = warp_incl_scan(d);
	const uint32_t ct = __shfl_sync(kFull, ci, 31);
	uint32_t b = 0;
	if (lane >= 30) b = atomicAdd(cnt + (lane - 30), lane == 30 ? ct : di);
	uint32_t pos = __shfl_sync(kFull, b, 30) + ci - c, off = __shfl_sync(kFull, b, 31) + di - d;
#pragma unroll
	for (int q = 0; q < Q; ++q) {
		const uint32_t dq = ok[q] ? deg[q] : 0u;
		if (ok[q]) {
			l.u[pos] = v[q];
			l.fb[pos] = beg[q] - off;
		}
		const bool wide = dq > 8;
		if (!wide)
			for (uint32_t i = off; i < min(off + dq, kSoloCap); ++i) l.owner[i] = (uint16_t) pos;
		for (uint32_t m = __ballot_sync(kFull, wide); m; m &= m - 1) {
			const int j = __ffs(m) - 1;
			const uint32_t jo = __shfl_sync(kFull, off, j), jd = __shfl_sync(kFull, dq, j), jp = __shfl_sync(kFull, pos, j);
			const uint32_t je = jo >= kSoloCap ? jo : jo + min(jd, kSoloCap - jo);
			for (uint32_t i = jo + lane; i < je; i += 32) l.owner[i] = (uint16_t) jp;
		}
		pos += ok[q];
		off += dq;
	}
}

// Expands the list `cur` (ne out-edges) into `nxt`, Q edges per lane in
// flight.  vis_s (may be null): the visited bits in shared memory.  The claim
// and the out-edge range of its vertex, whether it wins or
// not, go out together: two round trips per edge.
template <int Q, int kThreads>
__device__ __forceinline__ void solo_expand(const DevGraph &g, const RunCtx &r, const SoloList &cur, const SoloList &nxt,
		uint32_t *cn, uint32_t ne, int32_t nl, uint32_t *vis_s) {
	const unsigned lane = lane_id();
	for (uint32_t f0 = threadIdx.x - lane; f0 < ne; f0 += Q * kThreads) {
		bool ok[Q];
		uint32_t u[Q], v[Q], beg[Q], end[Q];
		int32_t old[Q];
#pragma unroll
		for (int q = 0; q < Q; ++q) {
			const uint32_t f = f0 + q * kThreads + lane;
			ok[q] = f < ne;
			const uint32_t j = ok[q] ? cur.owner[f] : 0u;
			u[q] = ok[q] ? cur.u[j] : 0u;
			v[q] = ok[q] ? __ldg(g.col + (cur.fb[j] + f)) : 0u;
		}
#pragma unroll
		for (int q = 0; q < Q; ++q) {
			beg[q] = ok[q] ? __ldg(g.row_off + v[q]) : 0u;
			end[q] = ok[q] ? __ldg(g.row_off + v[q] + 1) : 0u;
			const uint32_t bit = 1u << (v[q] & 31);
			if (!ok[q]) old[q] = 0;
			else if (vis_s) old[q] = (atomicOr(vis_s + (v[q] >> 5), bit) & bit) ? 0 : -1;
			else old[q] = atomicCAS((int *) r.level + v[q], -1, nl);
		}
#pragma unroll
		for (int q = 0; q < Q; ++q) {
			ok[q] = ok[q] && old[q] == -1;
			end[q] -= beg[q];
			if (ok[q]) {
				if (vis_s) r.level[v[q]] = nl;
				if (r.vis) atomicOr(r.vis + (v[q] >> 5), 1u << (v[q] & 31));
				if (r.parent) r.parent[v[q]] = u[q];
			}
		}
		solo_append<Q>(nxt, cn, ok, v, beg, end);
	}
}

} // namespace bfsg
