// build_device.cu -- the graph layout built on the GPU from an edge list:
// CSR, the in-edge lists and the packed column-major segments, by histogram,
// exclusive-scan and scatter kernels.
//
// It replaces, for large in-memory graphs, the host passes of the loader (the
// bucketing that tools/csr_tiling and tools/column_major_tile do,
// tools/csr_tiling/page_rank.cpp:531-567, tools/column_major_tile/kcore.cpp:
// 378-415, and this library's packing).  The scatters use atomics, so the
// order of edges inside a CSR row, an in-edge list or a packed segment is not
// the files' order; no traversal result depends on that order (levels are
// distances; parents are checked as a BFS tree).
#include <algorithm>
#include <cstdint>

#include "../../include/bfs_gb300.h"
#include "bc_batch.h"
#include "bfs_device.cuh"
#include "build_device.h"
#include "device_common.cuh"

namespace bfsg {

namespace {

constexpr int kBThreads = 512;
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;  // per thread
constexpr uint32_t kScanTile = kScanThreads * kScanItems;

__global__ void k_degrees(const uint32_t *src, const uint32_t *dst, uint64_t m, uint32_t n, uint32_t *out_deg,
		uint32_t *in_deg, int *err) {
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
		const uint32_t u = src[i], v = dst[i];
		if (u >= n || v >= n) {
			atomicExch(err, BFS_EFORMAT);
			continue;
		}
		atomicAdd(out_deg + u, 1u);
		atomicAdd(in_deg + v, 1u);
	}
}

// Block-wide exclusive scan of kScanTile values, in place in shared memory
// (thread t holds items 4t..4t+3).
__device__ void block_exclusive_scan(uint32_t *vals) {
	__shared__ uint32_t warp_tot[kScanThreads / 32];
	uint32_t v[kScanItems], sum = 0;
#pragma unroll
	for (int k = 0; k < kScanItems; ++k) {
		v[k] = vals[threadIdx.x * kScanItems + k];
		sum += v[k];
	}
	const uint32_t incl = warp_incl_scan(sum);
	if (lane_id() == 31) warp_tot[warp_id()] = incl;
	__syncthreads();
	if (warp_id() == 0) {
		const uint32_t t = lane_id() < kScanThreads / 32 ? warp_tot[lane_id()] : 0u;
		const uint32_t ti = warp_incl_scan(t);
		if (lane_id() < kScanThreads / 32) warp_tot[lane_id()] = ti - t;  // exclusive
	}
	__syncthreads();
	uint32_t run = warp_tot[warp_id()] + incl - sum;
#pragma unroll
	for (int k = 0; k < kScanItems; ++k) {
		vals[threadIdx.x * kScanItems + k] = run;
		run += v[k];
	}
	__syncthreads();
}

// Phase 1: the total of each tile.
__global__ void __launch_bounds__(kScanThreads) k_tile_sums(const uint32_t *in, uint32_t n, uint32_t *sums) {
	const uint64_t base = (uint64_t) blockIdx.x * kScanTile;
	uint32_t s = 0;
	for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads)
		if (base + k < n) s += in[base + k];
	s = warp_sum(s);
	__shared__ uint32_t ws[kScanThreads / 32];
	if (lane_id() == 0) ws[warp_id()] = s;
	__syncthreads();
	if (threadIdx.x == 0) {
		uint32_t t = 0;
		for (int w = 0; w < kScanThreads / 32; ++w) t += ws[w];
		sums[blockIdx.x] = t;
	}
}

// Phase 2 (one CTA): exclusive scan of the tile sums, in place; total at [tiles].
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(uint32_t *sums, uint32_t tiles) {
	__shared__ uint32_t buf[kScanTile];
	uint32_t carry = 0;
	for (uint32_t base = 0; base < tiles; base += kScanTile) {
		for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads) buf[k] = base + k < tiles ? sums[base + k] : 0u;
		__syncthreads();
		uint32_t last = buf[kScanTile - 1];
		__syncthreads();
		block_exclusive_scan(buf);
		for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads)
			if (base + k < tiles) sums[base + k] = buf[k] + carry;
		const uint32_t tile_total = buf[kScanTile - 1] + last;
		__syncthreads();
		carry += tile_total;
	}
	if (threadIdx.x == 0) sums[tiles] = carry;
}

// Phase 3: each tile's exclusive scan plus its offset; out[n] = total.
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const uint32_t *in, uint32_t n, const uint32_t *sums,
		uint32_t tiles, uint32_t *out) {
	__shared__ uint32_t buf[kScanTile];
	const uint64_t base = (uint64_t) blockIdx.x * kScanTile;
	for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads) buf[k] = base + k < n ? in[base + k] : 0u;
	__syncthreads();
	block_exclusive_scan(buf);
	const uint32_t off = sums[blockIdx.x];
	for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads)
		if (base + k < n) out[base + k] = buf[k] + off;
	if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = sums[tiles];
}

// out[pos] = val[i] with pos the next free slot of key[i]'s bucket.
__global__ void k_scatter(const uint32_t *key, const uint32_t *val, uint64_t m, uint32_t *cursor, uint32_t *out) {
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
		out[atomicAdd(cursor + key[i], 1u)] = val[i];
}

// Per vertex, from the degrees: the has-in-edge bitmap, the chunks of the
// batched pull (0 up to `big` in-edges) and whether there are any, the largest
// out-degree.
__global__ void k_vertex_facts(const uint32_t *out_deg, const uint32_t *in_deg, uint32_t n, uint32_t big, uint32_t chunk,
		uint32_t *hasin, uint32_t *chunks, uint32_t *is_big, uint32_t *max_degree) {
	const uint32_t stride = gridDim.x * blockDim.x;
	uint32_t mx = 0;
	for (uint32_t v0 = blockIdx.x * blockDim.x + threadIdx.x - lane_id(); v0 < n; v0 += stride) {
		const uint32_t v = v0 + lane_id();
		const uint32_t in = v < n ? in_deg[v] : 0u;
		const uint32_t bits = __ballot_sync(kFull, in != 0u);
		if (lane_id() == 0) hasin[v0 / 32] = bits;
		if (v >= n) continue;
		chunks[v] = in > big ? (in + chunk - 1) / chunk : 0u;
		is_big[v] = in > big;
		mx = max(mx, out_deg[v]);
	}
	__syncwarp();
	mx = __reduce_max_sync(kFull, mx);
	if (lane_id() == 0 && mx) atomicMax(max_degree, mx);
}

// Per vertex, the chunks of its list in batched betweenness (0 up to `chunk` edges).
__global__ void k_chunk_counts(const uint32_t *off, uint32_t n, uint32_t chunk, uint32_t *chunks) {
	const uint32_t stride = gridDim.x * blockDim.x;
	for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
		const uint32_t d = off[v + 1] - off[v];
		const uint32_t len = bb_chunk_len(chunk, d);
		chunks[v] = d > chunk ? d / len + (d % len != 0) : 0u;
	}
}

// The lists of the batched pull from the scans of chunks[] and is_big[]; without
// big_off the chunks of batched betweenness.
__global__ void k_big_lists(uint32_t n, const uint32_t *big_off, const uint32_t *chunk_off, const uint32_t *in_off,
		uint32_t nchunks, uint32_t chunk, uint32_t *in_big, uint32_t *chunk_v, uint32_t *chunk_beg) {
	const uint32_t stride = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
	for (uint32_t v = t; big_off && v < n; v += stride)
		if (big_off[v + 1] != big_off[v]) in_big[big_off[v]] = v;
	for (uint32_t c = t; c < nchunks; c += stride) {
		// the last vertex whose chunks start at or before c
		uint32_t lo = 0, hi = n;
		while (hi - lo > 1) {
			const uint32_t mid = lo + (hi - lo) / 2;
			if (chunk_off[mid] <= c) lo = mid;
			else hi = mid;
		}
		chunk_v[c] = lo;
		const uint32_t len = big_off ? chunk : bb_chunk_len(chunk, in_off[lo + 1] - in_off[lo]);
		chunk_beg[c] = in_off[lo] + (c - chunk_off[lo]) * len;
	}
}

// The non-empty blocks of the has-in-edge bitmap (one CTA, 1024 blocks at a time).
constexpr int kPbThreads = 1024;
__global__ void __launch_bounds__(kPbThreads) k_pull_blocks(const uint32_t *hasin, uint32_t nwords, uint32_t *blocks,
		uint32_t *count) {
	__shared__ uint32_t s_cnt[2][kPbThreads / 32];
	const uint32_t nb = (nwords + kPullBlock - 1) / kPullBlock;
	uint32_t run = 0, turn = 0;
	for (uint64_t b0 = 0; b0 < nb; b0 += kPbThreads, turn ^= 1u) {
		const uint64_t w0 = (b0 + threadIdx.x) * kPullBlock;
		uint32_t bits = 0;
#pragma unroll
		for (uint32_t q = 0; q < kPullBlock; ++q) bits |= w0 + q < nwords ? __ldg(hasin + w0 + q) : 0u;
		const uint32_t m = __ballot_sync(kFull, bits);
		if (lane_id() == 0) s_cnt[turn][warp_id()] = __popc(m);
		__syncthreads();
		const uint32_t c = s_cnt[turn][lane_id()];
		const uint32_t incl = warp_incl_scan(c);
		const uint32_t at = run + __shfl_sync(kFull, incl - c, warp_id()) + __popc(m & lanemask_lt());
		if (bits) blocks[at] = (uint32_t) b0 + threadIdx.x;
		run += __shfl_sync(kFull, incl, 31);
	}
	if (threadIdx.x == 0) *count = run;
}

// In-edges per tile column: the in-edge lists of a column are one range.
__global__ void k_col_edges(const uint32_t *in_off, uint32_t n, uint32_t w, uint32_t side, uint32_t *col_edges) {
	const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c < side) col_edges[c] = in_off[(uint32_t) min((uint64_t) (c + 1) * w, (uint64_t) n)] - in_off[c * w];
}

// ---- packed segments from the in-edge lists --------------------------------
// A column group is a destination range, so its edges are one range of the
// in-edge lists: a CTA takes up to kSegItem of them, counts them by stripe in
// shared memory, and goes to the segments' global counters once per stripe
// instead of once per edge.  (Pokec shape, 30.6 M edges: one global atomic per
// edge took 0.33 ms to count and 0.57 ms to fill.)
constexpr uint32_t kSegItem = 32768;
constexpr uint32_t kSegMaxStripes = 12288;  // 48 KB of counters
constexpr int kSegThreads = 1024;

__device__ __forceinline__ void seg_item_count(const uint32_t *in_src, const SegItem &it, uint32_t sw, uint32_t stripes,
		uint32_t *s_cnt) {
	for (uint32_t k = threadIdx.x; k < stripes; k += blockDim.x) s_cnt[k] = 0;
	__syncthreads();
	// (counted from the item's start: edge numbers go up to 2^32 - 1)
	for (uint32_t i = threadIdx.x; i < it.end - it.beg; i += blockDim.x)
		atomicAdd(s_cnt + __ldg(in_src + it.beg + i) / sw, 1u);
	__syncthreads();
}

__global__ void __launch_bounds__(kSegThreads) k_seg_count(const uint32_t *in_src, const SegItem *items, uint32_t sw,
		uint32_t stripes, uint32_t *seg_count) {
	extern __shared__ uint32_t s_cnt[];
	const SegItem it = items[blockIdx.x];
	seg_item_count(in_src, it, sw, stripes, s_cnt);
	for (uint32_t k = threadIdx.x; k < stripes; k += blockDim.x)
		if (s_cnt[k]) atomicAdd(seg_count + (size_t) it.group * stripes + k, s_cnt[k]);
}

// Packs the item's edges (the word layout of pack_tiles).  A warp takes a run
// of consecutive edges and walks the destinations' offsets along with it.
__global__ void __launch_bounds__(kSegThreads) k_seg_pack(const uint32_t *in_off, const uint32_t *in_src,
		const SegItem *items, DeviceBuildShape sh, uint32_t stripes, const uint32_t *group_col, uint32_t n,
		uint32_t *cursor, uint32_t *words) {
	extern __shared__ uint32_t s_cnt[];
	const SegItem it = items[blockIdx.x];
	const uint32_t sw = sh.s * sh.w;
	seg_item_count(in_src, it, sw, stripes, s_cnt);
	for (uint32_t k = threadIdx.x; k < stripes; k += blockDim.x)
		if (s_cnt[k]) s_cnt[k] = atomicAdd(cursor + (size_t) it.group * stripes + k, s_cnt[k]);
	__syncthreads();
	const uint32_t c0 = group_col[it.group], vend = (uint32_t) min((uint64_t) group_col[it.group + 1] * sh.w, (uint64_t) n);
	const uint32_t cshift = sh.vbits, ushift = sh.vbits + sh.cbits;
	const unsigned lane = lane_id(), nw = blockDim.x / 32;
	const uint32_t len = it.end - it.beg, per = ((len + nw - 1) / nw + 31) / 32 * 32;
	const uint32_t i0 = min(len, warp_id() * per), i1 = min(len, i0 + per), lo = it.beg + i0;
	if (i0 >= i1) return;
	// the last destination whose list starts at or before lo
	uint32_t vb = c0 * sh.w, vh = vend;
	while (vh - vb > 1) {
		const uint32_t mid = vb + (vh - vb) / 2;
		if (__ldg(in_off + mid) <= lo) vb = mid;
		else vh = mid;
	}
	for (uint32_t i = i0; i < i1; i += 32) {
		const bool mine = i + lane < i1;
		const uint32_t e = it.beg + i + lane;
		uint32_t v = 0;
		bool have = !mine;
		for (;;) {  // 32 destinations at a time until every lane has its own
			const uint32_t off = vb + lane + 1 <= vend ? __ldg(in_off + vb + lane + 1) : 0xFFFFFFFFu;  // ends of vb + lane
			uint32_t o = 0;  // lists of the 32 that end at or before e
#pragma unroll
			for (uint32_t st = 16; st; st >>= 1) {
				const uint32_t x = __shfl_sync(kFull, off, o + st - 1);
				if (x <= e) o += st;
			}
			const uint32_t lastoff = __shfl_sync(kFull, off, 31);
			const bool here = !have && lastoff > e;
			if (here) {
				v = vb + o;
				have = true;
			}
			if (__all_sync(kFull, have)) break;
			vb += 32;
		}
		if (mine) {
			const uint32_t u = __ldg(in_src + e), k = u / sw, c = v / sh.w;
			words[atomicAdd(s_cnt + k, 1u)] = (v - c * sh.w) | ((c - c0) << cshift) | ((u - k * sw) << ushift);
		}
		// the next 32 edges start at or after this run's last destination
		vb = __shfl_sync(kFull, v, 31 - __clz(__ballot_sync(kFull, mine)));
	}
}

__device__ __forceinline__ uint32_t seg_of(uint32_t u, uint32_t v, const DeviceBuildShape &sh, const uint32_t *group_of) {
	return group_of[v / sh.w] * sh.stripes + u / sh.w / sh.s;
}

__global__ void k_seg_hist(const uint32_t *src, const uint32_t *dst, uint64_t m, DeviceBuildShape sh,
		const uint32_t *group_of, uint32_t *seg_count) {
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
		atomicAdd(seg_count + seg_of(src[i], dst[i], sh, group_of), 1u);
}

// Packs u->v into its segment (the word layout of pack_tiles).
__global__ void k_seg_fill(const uint32_t *src, const uint32_t *dst, uint64_t m, DeviceBuildShape sh,
		const uint32_t *group_of, const uint32_t *group_col, uint32_t *cursor, uint32_t *words) {
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	const uint32_t cshift = sh.vbits, ushift = sh.vbits + sh.cbits;
	for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
		const uint32_t u = src[i], v = dst[i];
		const uint32_t k = u / sh.w / sh.s, c = v / sh.w, gi = group_of[c];
		const uint32_t word = (v - c * sh.w) | ((c - group_col[gi]) << cshift) | ((u - k * sh.s * sh.w) << ushift);
		words[atomicAdd(cursor + gi * sh.stripes + k, 1u)] = word;
	}
}

// Padding words after every segment's edges, up to the next segment.
__global__ void k_seg_pad(const uint32_t *seg_off, const uint32_t *seg_count, uint64_t nseg, uint32_t stripes,
		const uint32_t *pad_word, uint32_t *words) {
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	for (uint64_t j = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; j < nseg; j += stride) {
		const uint32_t pw = pad_word[j / stripes];
		for (uint32_t x = seg_off[j] + seg_count[j]; x < seg_off[j + 1]; ++x) words[x] = pw;
	}
}

int grid_for(uint64_t work, int num_sms) {
	const uint64_t g = (work + kBThreads - 1) / kBThreads;
	return (int) std::max<uint64_t>(1, std::min<uint64_t>(g, (uint64_t) num_sms * 8));
}

} // namespace

int dbuild_degrees(const uint32_t *src, const uint32_t *dst, uint64_t m, uint32_t n, uint32_t *out_deg,
		uint32_t *in_deg, int *err, int num_sms, cudaStream_t st) {
	k_degrees<<<grid_for(m, num_sms), kBThreads, 0, st>>>(src, dst, m, n, out_deg, in_deg, err);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

uint32_t dbuild_scan_tmp_words(uint32_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

int dbuild_exclusive_scan(const uint32_t *in, uint32_t n, uint32_t *tmp, uint32_t *out, cudaStream_t st) {
	const uint32_t tiles = dbuild_scan_tmp_words(n) - 1;
	if (tiles == 0) return cudaMemsetAsync(out, 0, sizeof(uint32_t), st) == cudaSuccess ? BFS_OK : BFS_ECUDA;
	k_tile_sums<<<tiles, kScanThreads, 0, st>>>(in, n, tmp);
	k_scan_sums<<<1, kScanThreads, 0, st>>>(tmp, tiles);
	k_scan_tiles<<<tiles, kScanThreads, 0, st>>>(in, n, tmp, tiles, out);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_scatter(const uint32_t *key, const uint32_t *val, uint64_t m, uint32_t *cursor, uint32_t *out, int num_sms,
		cudaStream_t st) {
	k_scatter<<<grid_for(m, num_sms), kBThreads, 0, st>>>(key, val, m, cursor, out);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_vertex_facts(const uint32_t *out_deg, const uint32_t *in_deg, uint32_t n, uint32_t big, uint32_t chunk,
		uint32_t *hasin, uint32_t *chunks, uint32_t *is_big, uint32_t *max_degree, int num_sms, cudaStream_t st) {
	k_vertex_facts<<<grid_for(n, num_sms), kBThreads, 0, st>>>(out_deg, in_deg, n, big, chunk, hasin, chunks, is_big,
			max_degree);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_chunk_counts(const uint32_t *off, uint32_t n, uint32_t chunk, uint32_t *chunks, int num_sms, cudaStream_t st) {
	k_chunk_counts<<<grid_for(n, num_sms), kBThreads, 0, st>>>(off, n, chunk, chunks);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_big_lists(uint32_t n, const uint32_t *big_off, const uint32_t *chunk_off, const uint32_t *in_off,
		uint32_t nchunks, uint32_t chunk, uint32_t *in_big, uint32_t *chunk_v, uint32_t *chunk_beg, int num_sms,
		cudaStream_t st) {
	k_big_lists<<<grid_for(n, num_sms), kBThreads, 0, st>>>(n, big_off, chunk_off, in_off, nchunks, chunk, in_big, chunk_v,
			chunk_beg);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_pull_blocks(const uint32_t *hasin, uint32_t nwords, uint32_t *blocks, uint32_t *count, cudaStream_t st) {
	static_assert(kPbThreads == 32 * 32, "a count per lane");
	k_pull_blocks<<<1, kPbThreads, 0, st>>>(hasin, nwords, blocks, count);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_col_edges(const uint32_t *in_off, uint32_t n, uint32_t w, uint32_t side, uint32_t *col_edges, cudaStream_t st) {
	k_col_edges<<<(side + kBThreads - 1) / kBThreads, kBThreads, 0, st>>>(in_off, n, w, side, col_edges);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

bool dbuild_seg_items_fit(uint32_t stripes) { return stripes <= kSegMaxStripes; }

std::vector<SegItem> dbuild_seg_items(const std::vector<uint32_t> &group_col, const std::vector<uint64_t> &col_edges) {
	std::vector<SegItem> items;
	uint64_t e = 0;
	for (uint32_t gi = 0; gi + 1 < group_col.size(); ++gi) {
		uint64_t end = e;
		for (uint32_t c = group_col[gi]; c < group_col[gi + 1]; ++c) end += col_edges[c];
		for (; e < end; e += std::min<uint64_t>(kSegItem, end - e))
			items.push_back({gi, (uint32_t) e, (uint32_t) std::min<uint64_t>(end, e + kSegItem)});
	}
	return items;
}

int dbuild_seg_count(const uint32_t *in_src, const SegItem *items, uint32_t num_items, uint32_t sw, uint32_t stripes,
		uint32_t *seg_count, cudaStream_t st) {
	if (!num_items) return BFS_OK;
	k_seg_count<<<num_items, kSegThreads, stripes * 4, st>>>(in_src, items, sw, stripes, seg_count);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_seg_pack(const uint32_t *in_off, const uint32_t *in_src, const SegItem *items, uint32_t num_items,
		const DeviceBuildShape &sh, const uint32_t *group_col, uint32_t n, uint32_t *cursor, uint32_t *words, cudaStream_t st) {
	if (!num_items) return BFS_OK;
	k_seg_pack<<<num_items, kSegThreads, sh.stripes * 4, st>>>(in_off, in_src, items, sh, sh.stripes, group_col, n, cursor,
			words);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_seg_hist(const uint32_t *src, const uint32_t *dst, uint64_t m, const DeviceBuildShape &sh,
		const uint32_t *group_of, uint32_t *seg_count, int num_sms, cudaStream_t st) {
	k_seg_hist<<<grid_for(m, num_sms), kBThreads, 0, st>>>(src, dst, m, sh, group_of, seg_count);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_seg_fill(const uint32_t *src, const uint32_t *dst, uint64_t m, const DeviceBuildShape &sh,
		const uint32_t *group_of, const uint32_t *group_col, uint32_t *cursor, uint32_t *words, int num_sms,
		cudaStream_t st) {
	k_seg_fill<<<grid_for(m, num_sms), kBThreads, 0, st>>>(src, dst, m, sh, group_of, group_col, cursor, words);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int dbuild_seg_pad(const uint32_t *seg_off, const uint32_t *seg_count, uint64_t nseg, uint32_t stripes,
		const uint32_t *pad_word, uint32_t *words, int num_sms, cudaStream_t st) {
	k_seg_pad<<<grid_for(nseg, num_sms), kBThreads, 0, st>>>(seg_off, seg_count, nseg, stripes, pad_word, words);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

} // namespace bfsg
