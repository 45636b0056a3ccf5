// bc.cu -- betweenness-centrality dependencies of one source, on the device.
//
// The reference's BC() (apps/betweennessCentrality_simd/bc.cpp:1717-2097)
// runs a forward BFS that adds path counts along every edge into a newly
// reached vertex (BFS_kernel_sparse :572-775, bfs_kernel_dense :1083-1162),
// keeps every level's frontier, then walks the frontiers backwards adding
// 1/paths to each vertex and pushing its sum to unvisited in-neighbours over
// the reverse graph (:1987-2030), and finally turns the sums into
// dependencies (:2032-2061).
//
// Here the levels come from the single-source traversal (k_bfs_persistent),
// and one cooperative launch does the rest with pulls instead of pushes (but
// for some of the integer path counts), so that every float sum has a fixed
// order:
//   1. level sort: reached vertices are ordered by (level, class), with the
//      vertices whose in- or out-degree exceeds kBcBig first in each level.
//      Each warp owns a range of 32*q vertices and counts / places them with
//      __match_any_sync, so the order is deterministic.
//   2. path counts, level by level: sigma(v) = sum of sigma(u) over in-edges
//      u -> v with level(u) = level(v) - 1 (unsigned, wraps like the
//      reference's unsigned adds).
//   3. dependency sums, deepest level first: D(v) = 1/sigma(v) + sum of D(w)
//      over out-edges v -> w with level(w) = level(v) + 1; the output is
//      (D - 1/sigma) / (1/sigma), 0 where sigma is 0 -- the reference's float
//      formulas, with its signed int -> float conversion of the counts.
// Per level, the edge lists of big vertices are cut into kBcWarpChunk-edge chunks
// that warps all over the grid sum (kBcChunk and CTAs where a level has very many
// big vertices; partials are added in chunk order by whoever completes the last
// one), medium vertices are summed by half-warps, and small
// ones by a lane each, with lanes of a warp in the same degree band.  Path
// counts of levels that few edges lead to are pushed instead (integer adds).
#include "bc.h"

#include <algorithm>
#include <type_traits>

#include "../../include/bfs_gb300.h"
#include "device_common.cuh"

namespace bfsg {
namespace {

constexpr int kBcThreads = 512;
constexpr int kBcWarps = kBcThreads / 32;
constexpr int kBcUnroll = 4;
constexpr uint32_t kBcSmemKeys = 256;  // level sort: keys a warp counts in shared memory

struct BcShared {
	float f[kBcWarps];
	uint32_t u[kBcWarps];
	unsigned long long e[kBcWarps];
	uint32_t scan[kBcWarps];
	uint32_t total;
	uint32_t chunk_beg, chunk_end;
	uint32_t beg[kBcClasses + 1];        // the level's classes in `order`
	uint32_t items[kBcClasses + 1];      // work items before each class
	uint32_t per[kBcClasses];            // vertices per item
	uint32_t lv_deg[2][kBcTraceLevels];  // this CTA's out- and in-degree sums by level
	union {
		uint32_t cpre[kBcSmemBig + 1];        // chunk prefix of the level's big vertices
		uint32_t keys[kBcWarps * kBcSmemKeys];  // level sort: a warp's counters
	};
};
__device__ __shared__ BcShared bsh;

template <class T> __device__ __forceinline__ T *bsh_slot();
template <> __device__ __forceinline__ float *bsh_slot<float>() { return bsh.f; }
template <> __device__ __forceinline__ uint32_t *bsh_slot<uint32_t>() { return bsh.u; }
template <> __device__ __forceinline__ unsigned long long *bsh_slot<unsigned long long>() { return bsh.e; }

// CTA-wide sum with a fixed association (all threads call; warp 0 gets it).
template <class T> __device__ __forceinline__ T block_sum(T x) {
	T *slot = bsh_slot<T>();
	x = warp_sum(x);
	if (lane_id() == 0) slot[warp_id()] = x;
	__syncthreads();
	T t = T(0);
	if (warp_id() == 0) {
		t = lane_id() < (unsigned) kBcWarps ? slot[lane_id()] : T(0);
		t = warp_sum(t);
	}
	__syncthreads();
	return t;
}

// CTA-wide exclusive scan; *total gets the CTA's sum (all threads call).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t *total) {
	const unsigned lane = lane_id(), wid = warp_id();
	const uint32_t incl = warp_incl_scan(x);
	if (lane == 31) bsh.scan[wid] = incl;
	__syncthreads();
	if (wid == 0) {
		const uint32_t w = lane < (unsigned) kBcWarps ? bsh.scan[lane] : 0u;
		const uint32_t wi = warp_incl_scan(w);
		if (lane < (unsigned) kBcWarps) bsh.scan[lane] = wi - w;
		if (lane == 31) bsh.total = wi;
	}
	__syncthreads();
	const uint32_t r = incl - x + bsh.scan[wid];
	*total = bsh.total;
	__syncthreads();
	return r;
}

// Sort key of a vertex: kBcClasses*level + class by the larger of its in- and
// out-degree d (0: d > 1024; 1..5: d in (512, 1024], (256, 512], (128, 256],
// (64, 128], (32, 64]; 6: d in (8, 32]; 7: d <= 8); -1 for unreached and
// out-of-range ids.
__device__ __forceinline__ int vertex_key(const BcArgs &a, uint64_t v, uint32_t depth, int *bad) {
	if (v >= a.n) return -1;
	const int lv = a.level[v];
	if (lv < 0) return -1;
	if ((uint32_t) lv > depth) { *bad = 1; return -1; }
	const uint32_t od = a.row_off[v + 1] - a.row_off[v];
	const uint32_t id = a.in_off[v + 1] - a.in_off[v];
	const uint32_t dmax = od > id ? od : id;
	int cls = (int) kBcClasses - 1;
	if (dmax > kBcTiny && dmax <= kBcMedium) cls = (int) kBcClasses - 2;
	if (dmax > kBcBig) cls = 0;
	else if (dmax > kBcMedium) cls = 1 + (31 - __clz(kBcBig - 1)) - (31 - __clz(dmax - 1));
	return (int) kBcClasses * lv + cls;
}

template <bool kFwd> struct Dir {
	using T = typename std::conditional<kFwd, uint32_t, float>::type;
	static __device__ __forceinline__ uint32_t bits(T x);
	static __device__ __forceinline__ const uint32_t *off(const BcArgs &a) { return kFwd ? a.in_off : a.row_off; }
	static __device__ __forceinline__ const uint32_t *adj(const BcArgs &a) { return kFwd ? a.in_src : a.col; }
	static __device__ __forceinline__ T value(uint32_t bits);
};
template <> __device__ __forceinline__ uint32_t Dir<true>::value(uint32_t bits) { return bits; }
template <> __device__ __forceinline__ float Dir<false>::value(uint32_t bits) { return __uint_as_float(bits); }
template <> __device__ __forceinline__ uint32_t Dir<true>::bits(uint32_t x) { return x; }
template <> __device__ __forceinline__ uint32_t Dir<false>::bits(float x) { return __float_as_uint(x); }

// {level, value} of a neighbour in one 8-byte load.  Where the level is the one
// asked for, the pair was written in an earlier phase; others' values may be
// being written and are not used.
__device__ __forceinline__ uint2 ld_lvx(const uint2 *p) { return ld_phase(p); }

// Level tags and value bits of the neighbours nb[] (0xFFFFFFFF: none): with
// use8 the byte level first and the value only where it matches `target`,
// else {level, value} in one 8-byte load.
template <int U>
__device__ __forceinline__ void gather_tags(const BcArgs &a, const uint32_t (&nb)[U], uint2 (&lx)[U], bool use8,
		int target) {
#pragma unroll
	for (int k = 0; k < U; ++k) {
		if (nb[k] == 0xFFFFFFFFu) lx[k] = make_uint2(0xFFFFFFFEu, 0u);
		else if (use8) lx[k] = make_uint2((uint32_t) ld_cg_u8(a.lv8 + nb[k]), 0u);
		else lx[k] = ld_lvx(a.lvx + nb[k]);
	}
	if (use8) {
#pragma unroll
		for (int k = 0; k < U; ++k)
			if ((int) lx[k].x == target) lx[k].y = ld_cg(reinterpret_cast<const uint32_t *>(a.lvx + nb[k]) + 1);
	}
}

// Sum over the edges [beg, end) of one vertex by the whole CTA (result in warp 0).
template <bool kFwd>
__device__ __forceinline__ typename Dir<kFwd>::T cta_range_sum(const BcArgs &a, uint64_t beg, uint64_t end, int target,
		bool use8) {
	using T = typename Dir<kFwd>::T;
	const uint32_t *adj = Dir<kFwd>::adj(a);
	T s = T(0);
	for (uint64_t e = beg + threadIdx.x; e < end; e += (uint64_t) kBcThreads * kBcUnroll) {
		uint32_t nb[kBcUnroll];
		uint2 lx[kBcUnroll];
#pragma unroll
		for (int k = 0; k < kBcUnroll; ++k) {
			const uint64_t ee = e + (uint64_t) k * kBcThreads;
			nb[k] = ee < end ? __ldg(adj + ee) : 0xFFFFFFFFu;
		}
		gather_tags(a, nb, lx, use8, target);
#pragma unroll
		for (int k = 0; k < kBcUnroll; ++k)
			if ((int) lx[k].x == target) s += Dir<kFwd>::value(lx[k].y);
	}
	return block_sum(s);
}


// Chunk prefix of the vertices order[bb .. bb+cnt) (cnt <= kBcSmemBig, `per`
// edges per chunk, `least` chunks or more each) in bsh.cpre, the same in every
// CTA; returns the total.
template <bool kFwd>
__device__ __forceinline__ uint32_t chunk_prefix(const BcArgs &a, uint32_t bb, uint32_t cnt, uint32_t per, uint32_t least) {
	const uint32_t *off = Dir<kFwd>::off(a);
	constexpr uint32_t kPer = kBcSmemBig / kBcThreads;  // consecutive entries per thread, their loads together
	uint32_t v[kPer], c[kPer], sum = 0;
#pragma unroll
	for (uint32_t k = 0; k < kPer; ++k) {
		const uint32_t i = threadIdx.x * kPer + k;
		v[k] = i < cnt ? ld_cg(a.order + bb + i) : 0xFFFFFFFFu;
	}
#pragma unroll
	for (uint32_t k = 0; k < kPer; ++k) {
		c[k] = v[k] != 0xFFFFFFFFu ? max(least, (off[v[k] + 1] - off[v[k]] + per - 1) / per) : 0u;
		sum += c[k];
	}
	uint32_t total;
	uint32_t run = block_excl_scan(sum, &total);
#pragma unroll
	for (uint32_t k = 0; k < kPer; ++k) {
		const uint32_t i = threadIdx.x * kPer + k;
		if (i < cnt) bsh.cpre[i] = run;
		run += c[k];
	}
	if (threadIdx.x == 0) bsh.cpre[cnt] = total;
	__syncthreads();
	return total;
}
// The largest i with cpre[i] <= j (cpre[cnt] > j).
__device__ __forceinline__ uint32_t chunk_owner(uint32_t cnt, uint32_t j) {
	uint32_t lo = 0, hi = cnt;
	while (lo < hi) {
		const uint32_t mid = (lo + hi + 1) / 2;
		if (bsh.cpre[mid] <= j) lo = mid;
		else hi = mid - 1;
	}
	return lo;
}

template <bool kFwd>
__device__ __forceinline__ typename Dir<kFwd>::T big_finish_sum(const BcArgs &a, uint32_t i, bool global);

// Writes a vertex's finished sum (one thread).
template <bool kFwd> __device__ __forceinline__ void finish_vertex(const BcArgs &a, uint32_t v, typename Dir<kFwd>::T sum);

// Chunk j (kBcWarpChunk edges) of the level's big vertices order[bb .. bb+nbig)
// (prefix in bsh.cpre) by one warp, into partial[j] (value bits); the warp
// that completes a vertex's last chunk adds them in a fixed order and writes
// the vertex, and leaves its count at 0.
template <bool kFwd>
__device__ __forceinline__ void big_chunk(const BcArgs &a, uint32_t bb, uint32_t nbig, uint32_t j, int target, bool use8,
		unsigned long long *edges) {
	using T = typename Dir<kFwd>::T;
	const uint32_t *off = Dir<kFwd>::off(a), *adj = Dir<kFwd>::adj(a);
	const uint32_t lo = chunk_owner(nbig, j), c0 = bsh.cpre[lo], c1 = bsh.cpre[lo + 1];
	const uint32_t v = ld_cg(a.order + bb + lo);
	const uint32_t vbeg = off[v], vend = off[v + 1];
	const uint32_t beg = vbeg + (j - c0) * kBcWarpChunk, len = min(kBcWarpChunk, vend - beg);
	T s = T(0);
	for (uint32_t i = lane_id(); i < len; i += 32 * kBcUnroll) {
		uint32_t nb[kBcUnroll];
		uint2 lx[kBcUnroll];
#pragma unroll
		for (int k = 0; k < kBcUnroll; ++k) nb[k] = i + 32 * k < len ? __ldg(adj + beg + i + 32 * k) : 0xFFFFFFFFu;
		gather_tags(a, nb, lx, use8, target);
#pragma unroll
		for (int k = 0; k < kBcUnroll; ++k)
			if ((int) lx[k].x == target) s += Dir<kFwd>::value(lx[k].y);
	}
	__syncwarp();
	s = warp_sum(s);
	uint32_t before = 0;
	if (lane_id() == 0) {
		a.partial[j] = Dir<kFwd>::bits(s);
		// releases this partial to, and acquires the others' from, the chunks that count here
		asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(a.big_done + lo) : "memory");
	}
	if (__shfl_sync(kFull, before, 0) != c1 - c0 - 1) return;
	__syncwarp();
	const T t = big_finish_sum<kFwd>(a, lo, false);
	if (lane_id() == 0) {
		a.big_done[lo] = 0u;
		finish_vertex<kFwd>(a, v, t);
		*edges += vend - vbeg;
	}
}

// The same for a level with more than kBcSmemBig big vertices: the chunk
// prefix is scanned grid-wide into a.cpre (two grid barriers), then CTA c sums
// the contiguous chunk range [c*per, (c+1)*per).  Returns false when a barrier
// gave up.
template <bool kFwd>
__device__ __forceinline__ bool big_chunks_global(const BcArgs &a, uint32_t bb, uint32_t nbig, int target, bool use8,
		unsigned &epoch) {
	const uint32_t *off = Dir<kFwd>::off(a);
	BcControl *ctl = a.ctl;
	const uint32_t L = (nbig + gridDim.x - 1) / gridDim.x;
	const uint32_t lo = blockIdx.x * L < nbig ? blockIdx.x * L : nbig;
	const uint32_t hi = lo + L < nbig ? lo + L : nbig;
	{
		uint32_t s = 0;
		for (uint32_t i = lo + threadIdx.x; i < hi; i += kBcThreads) {
			const uint32_t v = ld_cg(a.order + bb + i);
			s += (off[v + 1] - off[v] + kBcChunk - 1) / kBcChunk;
		}
		s = block_sum(s);
		if (threadIdx.x == 0) ctl->blk[blockIdx.x] = s;
	}
	if (!grid_sync(ctl->bar, epoch, &ctl->err)) return false;
	uint32_t base = 0, total = 0;
	for (uint32_t c = threadIdx.x; c < gridDim.x; c += kBcThreads) {
		const uint32_t x = ld_cg(ctl->blk + c);
		if (c < blockIdx.x) base += x;
		total += x;
	}
	base = block_sum(base);
	total = block_sum(total);
	if (threadIdx.x == 0) {
		bsh.chunk_beg = base;
		bsh.chunk_end = total;
	}
	__syncthreads();
	base = bsh.chunk_beg;
	total = bsh.chunk_end;
	__syncthreads();
	for (uint32_t t0 = lo; t0 < hi; t0 += kBcThreads) {
		const uint32_t i = t0 + threadIdx.x;
		uint32_t c = 0;
		if (i < hi) {
			const uint32_t v = ld_cg(a.order + bb + i);
			c = (off[v + 1] - off[v] + kBcChunk - 1) / kBcChunk;
		}
		uint32_t tot;
		const uint32_t ex = block_excl_scan(c, &tot);
		if (i < hi) a.cpre[i] = base + ex;
		base += tot;
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) a.cpre[nbig] = total;
	if (!grid_sync(ctl->bar, epoch, &ctl->err)) return false;
	const uint32_t per = (total + gridDim.x - 1) / gridDim.x;
	const uint32_t j0 = blockIdx.x * per < total ? blockIdx.x * per : total;
	const uint32_t j1 = j0 + per < total ? j0 + per : total;
	uint32_t owner = 0;
	if (j0 < j1 && threadIdx.x == 0) {
		// the largest i with cpre[i] <= j0 (cpre[nbig] = total > j0)
		uint32_t l = 0, h = nbig;
		while (l < h) {
			const uint32_t mid = (l + h + 1) / 2;
			if (ld_cg(a.cpre + mid) <= j0) l = mid;
			else h = mid - 1;
		}
		owner = l;
	}
	for (uint32_t j = j0; j < j1; ++j) {
		if (threadIdx.x == 0) {
			while (ld_cg(a.cpre + owner + 1) <= j) ++owner;
			const uint32_t v = ld_cg(a.order + bb + owner);
			const uint32_t beg = off[v] + (j - ld_cg(a.cpre + owner)) * kBcChunk;
			const uint32_t end = off[v + 1];
			bsh.chunk_beg = beg;
			bsh.chunk_end = end - beg > kBcChunk ? beg + kBcChunk : end;
		}
		__syncthreads();
		const uint32_t beg = bsh.chunk_beg, end = bsh.chunk_end;
		const typename Dir<kFwd>::T s = cta_range_sum<kFwd>(a, beg, end, target, use8);
		if (threadIdx.x == 0) a.partial[j] = Dir<kFwd>::bits(s);
	}
	return true;
}

// Sum of big vertex i's chunk partials in chunk order, by one warp (all lanes
// get it); the chunk prefix is in shared memory (global: in a.cpre).
template <bool kFwd>
__device__ __forceinline__ typename Dir<kFwd>::T big_finish_sum(const BcArgs &a, uint32_t i, bool global) {
	using T = typename Dir<kFwd>::T;
	const uint32_t c0 = global ? ld_cg(a.cpre + i) : bsh.cpre[i];
	const uint32_t c1 = global ? ld_cg(a.cpre + i + 1) : bsh.cpre[i + 1];
	T s = T(0);
	for (uint32_t j = c0 + lane_id(); j < c1; j += 32) s += Dir<kFwd>::value(ld_cg(a.partial + j));
	return warp_sum(s);
}

// Sum over the edges [beg, end) of one vertex by a half-warp (16 lanes).  Both
// halves call it together (the reduction shuffles the warp).
template <bool kFwd>
__device__ __forceinline__ typename Dir<kFwd>::T half_vertex_sum(const BcArgs &a, uint32_t beg, uint32_t end, int target,
		bool use8) {
	using T = typename Dir<kFwd>::T;
	const uint32_t *adj = Dir<kFwd>::adj(a);
	const uint32_t hl = lane_id() & 15u;
	T s = T(0);
	for (uint32_t e = beg + hl; e < end; e += 16u * kBcUnroll) {
		uint32_t nb[kBcUnroll];
		uint2 lx[kBcUnroll];
#pragma unroll
		for (int k = 0; k < kBcUnroll; ++k) {
			const uint32_t ee = e + (uint32_t) k * 16u;
			nb[k] = ee < end ? __ldg(adj + ee) : 0xFFFFFFFFu;
		}
		gather_tags(a, nb, lx, use8, target);
#pragma unroll
		for (int k = 0; k < kBcUnroll; ++k)
			if ((int) lx[k].x == target) s += Dir<kFwd>::value(lx[k].y);
	}
#pragma unroll
	for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(kFull, s, d);
	return s;
}

// Sum over the edges [beg, end) of one vertex by one lane: the list in
// aligned 16-byte pieces, kBcQuads of them and their neighbours' values in
// flight.  (32 vertices' concatenated lists walked by the warp, with an owner
// search and a segmented scan per 32 edges, spent about 60 shuffles per 32
// edges: 0.11 ms for the 8 M edges of a Pokec-shape level.)
constexpr int kBcQuads = 2;
template <bool kFwd>
__device__ __forceinline__ typename Dir<kFwd>::T lane_vertex_sum(const BcArgs &a, uint32_t beg, uint32_t end, int target,
		bool use8) {
	using T = typename Dir<kFwd>::T;
	const uint32_t *adj = Dir<kFwd>::adj(a);
	T s = T(0), lost = T(0);
	const uint32_t from = beg & ~3u;
	for (uint32_t i = 0; i < end - from; i += 4 * kBcQuads) {
		const uint32_t q = from + i;
		uint32_t nb[4 * kBcQuads];
		uint2 lx[4 * kBcQuads];
#pragma unroll
		for (int k = 0; k < kBcQuads; ++k) {
			const uint32_t e = q + 4 * k;
			if (i + 4 * k >= end - from) {
				nb[4 * k] = nb[4 * k + 1] = nb[4 * k + 2] = nb[4 * k + 3] = 0xFFFFFFFFu;
			} else if (a.m - e >= 4) {
				const uint4 x = ldg_v4(adj + e);
				nb[4 * k] = e >= beg ? x.x : 0xFFFFFFFFu;
				nb[4 * k + 1] = e + 1 >= beg && e + 1 < end ? x.y : 0xFFFFFFFFu;
				nb[4 * k + 2] = e + 2 >= beg && e + 2 < end ? x.z : 0xFFFFFFFFu;
				nb[4 * k + 3] = e + 3 >= beg && e + 3 < end ? x.w : 0xFFFFFFFFu;
			} else {  // the last edges of the array
#pragma unroll
				for (uint32_t t = 0; t < 4; ++t) nb[4 * k + t] = e + t >= beg && e + t < end ? __ldg(adj + e + t) : 0xFFFFFFFFu;
			}
		}
		gather_tags(a, nb, lx, use8, target);
		// pairwise, and what is rounded off where the groups meet (Knuth's TwoSum)
		// is added at the end: a lane's sum is then as near as a warp's tree
		T x[4 * kBcQuads];
#pragma unroll
		for (int k = 0; k < 4 * kBcQuads; ++k) x[k] = (int) lx[k].x == target ? Dir<kFwd>::value(lx[k].y) : T(0);
#pragma unroll
		for (int d = 1; d < 4 * kBcQuads; d *= 2)
#pragma unroll
			for (int k = 0; k + d < 4 * kBcQuads; k += 2 * d) x[k] += x[k + d];
		if constexpr (kFwd) {
			s += x[0];
		} else {
			const T t = s + x[0], b = t - s;
			lost += (s - (t - b)) + (x[0] - b);
			s = t;
		}
	}
	if constexpr (kFwd) return s;
	// an infinite sum (path counts wrap on street grids, and their reciprocals add up
	// past the largest float) rounds nothing off: lost is NaN then
	else return s + (isfinite(lost) ? lost : T(0));
}

// Path counts of level d pushed along the out-edges of the vertices of level
// d - 1 (order[bb .. bb+cnt), cnt <= kBcSmemBig): integer adds, whose order does
// not matter.  Warps take chunks of kBcPushChunk edges.
constexpr uint32_t kBcPushChunk = 512;
__device__ __forceinline__ void push_paths(const BcArgs &a, uint32_t bb, uint32_t cnt, int target, bool use8,
		unsigned long long *edges) {
	const uint32_t total = chunk_prefix<false>(a, bb, cnt, kBcPushChunk, 0);
	const unsigned lane = lane_id();
	const uint32_t gw = blockIdx.x + warp_id() * gridDim.x, tw = gridDim.x * kBcWarps;
	for (uint32_t j = gw; j < total; j += tw) {
		const uint32_t lo = chunk_owner(cnt, j);
		const uint32_t u = ld_cg(a.order + bb + lo);
		const uint32_t beg = a.row_off[u] + (j - bsh.cpre[lo]) * kBcPushChunk;
		const uint32_t len = min(kBcPushChunk, a.row_off[u + 1] - beg);
		const uint32_t su = ld_cg(reinterpret_cast<const uint32_t *>(a.lvx + u) + 1);
		if (lane == 0) *edges += len;
		for (uint32_t i = lane; i < len; i += 32 * kBcUnroll) {
			uint32_t v[kBcUnroll], lv[kBcUnroll];
#pragma unroll
			for (int k = 0; k < kBcUnroll; ++k) v[k] = i + 32 * k < len ? __ldg(a.col + beg + i + 32 * k) : 0xFFFFFFFFu;
#pragma unroll
			for (int k = 0; k < kBcUnroll; ++k)
				lv[k] = v[k] == 0xFFFFFFFFu ? 0xFFFFFFFEu
						: use8 ? (uint32_t) ld_cg_u8(a.lv8 + v[k]) : ld_cg(reinterpret_cast<const uint32_t *>(a.lvx + v[k]));
#pragma unroll
			for (int k = 0; k < kBcUnroll; ++k)
				if ((int) lv[k] == target) atomicAdd(reinterpret_cast<uint32_t *>(a.lvx + v[k]) + 1, su);
		}
	}
}

// sg: the vertex's path count
__device__ __forceinline__ void finish_dependency(const BcArgs &a, uint32_t v, float sum, uint32_t sg) {
	const float inv = sg ? 1.0f / (float) (int) sg : 0.0f;
	const float dv = sum + inv;
	a.lvx[v].y = __float_as_uint(dv);
	const float del = inv != 0.0f ? (dv - inv) / inv : 0.0f;
	a.delta[v] = del;
	if (a.acc && v != a.source) a.acc[v] += del;
}

template <> __device__ __forceinline__ void finish_vertex<true>(const BcArgs &a, uint32_t v, uint32_t sum) {
	a.sigma[v] = sum;
	a.lvx[v].y = sum;
}
template <> __device__ __forceinline__ void finish_vertex<false>(const BcArgs &a, uint32_t v, float sum) {
	finish_dependency(a, v, sum, ld_cg(a.sigma + v));
}

// The vertices order[i], order[i + step], ... below `last`, one per half-warp
// (kHalf) or lane: their sums for a level (none of their edges with `skip`).
// The next vertex's edge range and path count and the one after's id are
// loaded while a vertex is summed: without that, the chain order -> offsets ->
// edges -> values -> count of each vertex is what a level waits for.
template <bool kFwd, bool kHalf>
__device__ __forceinline__ void sum_vertices(const BcArgs &a, uint32_t i, uint32_t step, uint32_t last, int target,
		bool skip, bool use8, unsigned long long *edges) {
	using T = typename Dir<kFwd>::T;
	const uint32_t *off = Dir<kFwd>::off(a);
	const bool writer = !kHalf || (lane_id() & 15u) == 0;
	auto id_at = [&](uint32_t k) { return k < last ? ld_cg(a.order + k) : 0xFFFFFFFFu; };
	uint32_t v = id_at(i), next = id_at(i + step);
	uint32_t beg = 0, end = 0, sg = 0;
	if (v != 0xFFFFFFFFu) {
		beg = off[v];
		end = off[v + 1];
		if (!kFwd && writer) sg = ld_cg(a.sigma + v);
	}
	while (__any_sync(kFull, v != 0xFFFFFFFFu)) {
		const uint32_t next2 = next != 0xFFFFFFFFu ? id_at(i + 2 * step) : 0xFFFFFFFFu;
		uint32_t nbeg = 0, nend = 0, nsg = 0;
		if (next != 0xFFFFFFFFu) {
			nbeg = off[next];
			nend = off[next + 1];
			if (!kFwd && writer) nsg = ld_cg(a.sigma + next);
		}
		T s = T(0);
		if (!skip) {
			if constexpr (kHalf) s = half_vertex_sum<kFwd>(a, beg, end, target, use8);
			else s = lane_vertex_sum<kFwd>(a, beg, end, target, use8);
		}
		if (writer && v != 0xFFFFFFFFu) {
			if constexpr (kFwd) finish_vertex<true>(a, v, s);
			else finish_dependency(a, v, s, sg);
			if (!skip) *edges += end - beg;
		}
		__syncwarp();
		v = next;
		next = next2;
		beg = nbeg;
		end = nend;
		sg = nsg;
		i += step;
	}
}

// Of cnt vertices of class c (1 .. kBcClasses - 1), how many a warp takes at a
// time: at most about 2048 edges' worth, fewer where that would leave less than
// two items per warp of the grid, at least one step's (a vertex per half-warp
// or lane).
__device__ __forceinline__ uint32_t class_item(uint32_t c, uint32_t cnt) {
	const uint32_t least = c + 2 < kBcClasses ? 2u : 32u;
	const uint32_t most = c + 2 < kBcClasses ? 1u << c : c + 2 == kBcClasses ? 128u : 256u;
	return least * max(1u, min(most / least, cnt / (least * 2 * gridDim.x * kBcWarps)));
}

// All vertices of level d: big ones in chunks (`big`: not done by
// big_chunks_global), then the medium bands, then the small ones, dealt to the
// grid's warps in turn.  (With a CTA per chunk of 4096 edges, warps spent 39%
// of their cycles at block barriers; handed out through a counter, small
// levels paid more for the claims than large ones gained.)  What bounds a large
// level is the L1 pipeline: a neighbour's pair is a 32-byte sector of its own
// (18 M in-edges of a Pokec-shape level in 0.10 ms, 0.6 a cycle and SM).
// `skip`: the level's sums are all empty.
template <bool kFwd>
__device__ __forceinline__ void level_sums(const BcArgs &a, uint32_t d, int target, bool big, bool skip, bool use8,
		unsigned long long *edges) {
	__syncthreads();
	if (threadIdx.x <= kBcClasses) bsh.beg[threadIdx.x] = ld_cg(a.kstart + kBcClasses * d + threadIdx.x);
	__syncthreads();
	const uint32_t bb = bsh.beg[0], nbig = bsh.beg[1] - bb;
	uint32_t chunks = 0;
	// a vertex is finished with its last chunk, so one that is big for its other
	// side's edges and has none on this side (a sink of many in-edges) has a chunk too
	if (big && nbig && !skip) chunks = chunk_prefix<kFwd>(a, bb, nbig, kBcWarpChunk, 1);
	if (threadIdx.x == 0) {
		uint32_t n = chunks;
		for (uint32_t c = 1; c < kBcClasses; ++c) {
			bsh.items[c] = n;
			const uint32_t cnt = bsh.beg[c + 1] - bsh.beg[c], per = class_item(c, cnt);
			bsh.per[c] = per;
			n += (cnt + per - 1) / per;
		}
		bsh.items[kBcClasses] = n;
	}
	__syncthreads();
	const unsigned lane = lane_id();
	if (skip)
		for (uint32_t i = blockIdx.x * kBcThreads + threadIdx.x; i < nbig; i += gridDim.x * kBcThreads)
			finish_vertex<kFwd>(a, ld_cg(a.order + bb + i), typename Dir<kFwd>::T(0));
	const uint32_t total = bsh.items[kBcClasses];
	// warps numbered across CTAs first, so that a few items are spread over all SMs
	const uint32_t step = gridDim.x * kBcWarps;
	uint32_t item = warp_id() * gridDim.x + blockIdx.x;
	for (; item < chunks; item += step) big_chunk<kFwd>(a, bb, nbig, item, target, use8, edges);
	for (; item < total; item += step) {
		uint32_t c = 1;
		while (item >= bsh.items[c + 1]) ++c;
		const uint32_t first = bsh.beg[c] + (item - bsh.items[c]) * bsh.per[c];
		const uint32_t last = min(first + bsh.per[c], bsh.beg[c + 1]);
		if (c + 2 < kBcClasses) sum_vertices<kFwd, true>(a, first + (lane >> 4), 2, last, target, skip, use8, edges);
		else sum_vertices<kFwd, false>(a, first + lane, 32, last, target, skip, use8, edges);
	}
}

__global__ void __launch_bounds__(kBcThreads, 2) k_bc(BcArgs a) {
	BcControl *ctl = a.ctl;
	const unsigned lane = lane_id();
	const uint32_t gw = blockIdx.x * kBcWarps + warp_id();
	const uint32_t tw = gridDim.x * kBcWarps;
	if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t[0] = global_timer_ns();
	// the traversal's outcome decides for every CTA alike
	const int bfs_st = *(const volatile int *) a.bfs_status;
	const uint32_t steps = *(const volatile uint32_t *) a.num_steps;
	if (bfs_st != 0 || steps == 0 || steps > kBcMaxLevels) {
		if (blockIdx.x == 0 && threadIdx.x == 0)
			ctl->err = bfs_st != 0 ? bfs_st : (steps == 0 ? BFS_ECUDA : BFS_EUNSUPPORTED);
		return;
	}
	const uint32_t depth = steps - 1;
	const bool use8 = a.byte_levels && depth <= 254;
	const uint32_t K = kBcClasses * steps;
	const uint64_t W32 = ((uint64_t) a.n + 31) / 32;
	uint64_t q = (K * W32 + kBcCntCap - 1) / kBcCntCap;
	if (q == 0) q = 1;
	uint64_t R = (W32 + q - 1) / q;
	while ((uint64_t) K * R > kBcCntCap) {
		++q;
		R = (W32 + q - 1) / q;
	}
	// few keys: ranges as long as a warp's share, counted in shared memory (one
	// range per 32 vertices has KR = 2.5 M scattered counters on the Pokec shape)
	const bool skeys = K <= kBcSmemKeys;
	if (skeys) {
		q = max(q, (W32 + tw - 1) / tw);
		R = (W32 + q - 1) / q;
	}
	uint32_t *my_cnt = bsh.keys + (skeys ? warp_id() * K : 0u);
	const uint64_t KR = (uint64_t) K * R;
	unsigned epoch = 0;
	for (uint32_t i = threadIdx.x; i < 2 * kBcTraceLevels; i += kBcThreads) bsh.lv_deg[i / kBcTraceLevels][i % kBcTraceLevels] = 0;
	__syncthreads();

	// ---- 1a. count (level key, range) and initialise the outputs ----------
	unsigned long long my_edges = 0;
	uint32_t my_reached = 0;
	int bad = 0;
	for (uint64_t r = gw; r < R; r += tw) {
		if (skeys) for (uint32_t k = lane; k < K; k += 32) my_cnt[k] = 0;
		else for (uint32_t k = lane; k < K; k += 32) a.cnt[(uint64_t) k * R + r] = 0;
		__syncwarp();
		const uint64_t v0 = r * 32 * q;
		for (uint64_t j = 0; j < q; ++j) {
			const uint64_t v = v0 + j * 32 + lane;
			const int key = vertex_key(a, v, depth, &bad);
			if (v < a.n) {
				a.sigma[v] = v == a.source ? 1u : 0u;
				if (v < kBcSmemBig) a.big_done[v] = 0u;
				a.delta[v] = 0.0f;
				const int lv = a.level[v];
				a.lvx[v] = make_uint2((uint32_t) lv, v == a.source ? 1u : 0u);
				a.lv8[v] = (uint8_t) (lv < 0 || lv > 254 ? 255 : lv);
			}
			if (key >= 0) {
				++my_reached;
				const uint32_t od = a.row_off[v + 1] - a.row_off[v];
				my_edges += od;
				const uint32_t lv = (uint32_t) key / kBcClasses;
				if (lv < kBcTraceLevels) {
					atomicAdd(&bsh.lv_deg[0][lv], od);
					atomicAdd(&bsh.lv_deg[1][lv], a.in_off[v + 1] - a.in_off[v]);
				}
			}
			const unsigned mm = __match_any_sync(kFull, key);
			if (key >= 0 && lane == (unsigned) (__ffs(mm) - 1)) {
				if (skeys) my_cnt[key] += __popc(mm);
				else a.cnt[(uint64_t) key * R + r] += __popc(mm);
			}
			__syncwarp();
		}
		if (skeys) for (uint32_t k = lane; k < K; k += 32) a.cnt[(uint64_t) k * R + r] = my_cnt[k];
		__syncwarp();
	}
	__syncthreads();
	if (threadIdx.x < 2 * kBcTraceLevels) {
		const uint32_t x = (&bsh.lv_deg[0][0])[threadIdx.x];
		if (x) atomicAdd(&ctl->lv_deg[0][0] + threadIdx.x, x);
	}
	{
		const unsigned long long e = block_sum(my_edges);
		const uint32_t rc = block_sum(my_reached);
		const uint32_t b = block_sum((uint32_t) bad);
		if (threadIdx.x == 0) {
			if (e) atomicAdd(&ctl->edges_reached, e);
			if (rc) atomicAdd(&ctl->reached, rc);
			if (b) atomicExch(&ctl->err, BFS_ECUDA);
		}
	}
	if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;

	// ---- 1b. exclusive scan of the counters (key-major) --------------------
	const uint64_t L = (KR + gridDim.x - 1) / gridDim.x;
	const uint64_t lo = (uint64_t) blockIdx.x * L < KR ? (uint64_t) blockIdx.x * L : KR;
	const uint64_t hi = lo + L < KR ? lo + L : KR;
	{
		uint32_t s = 0;
		for (uint64_t i = lo + threadIdx.x; i < hi; i += kBcThreads) s += a.cnt[i];
		s = block_sum(s);
		if (threadIdx.x == 0) ctl->blk[blockIdx.x] = s;
	}
	if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;
	{
		uint32_t base = 0;
		for (uint32_t c = threadIdx.x; c < blockIdx.x; c += kBcThreads) base += ld_cg(ctl->blk + c);
		base = block_sum(base);
		if (warp_id() == 0 && lane == 0) bsh.u[0] = base;
		__syncthreads();
		base = bsh.u[0];
		__syncthreads();
		for (uint64_t t0 = lo; t0 < hi; t0 += kBcThreads) {
			const uint64_t i = t0 + threadIdx.x;
			const uint32_t x = i < hi ? a.cnt[i] : 0u;
			uint32_t tot;
			const uint32_t ex = block_excl_scan(x, &tot) + base;
			if (i < hi) {
				a.cnt[i] = ex;
				if (i % R == 0) a.kstart[i / R] = ex;
			}
			base += tot;
		}
		if (blockIdx.x == 0 && threadIdx.x == 0) a.kstart[K] = ld_cg(&ctl->reached);
	}
	if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;

	// ---- 1c. place the vertices ------------------------------------------
	for (uint64_t r = gw; r < R; r += tw) {
		const uint64_t v0 = r * 32 * q;
		if (skeys) for (uint32_t k = lane; k < K; k += 32) my_cnt[k] = ld_cg(a.cnt + (uint64_t) k * R + r);
		__syncwarp();
		for (uint64_t j = 0; j < q; ++j) {
			const uint64_t v = v0 + j * 32 + lane;
			int dummy = 0;
			const int key = vertex_key(a, v, depth, &dummy);
			const unsigned mm = __match_any_sync(kFull, key);
			const unsigned leader = (unsigned) (__ffs(mm) - 1);
			uint32_t base = 0;
			if (key >= 0 && lane == leader) base = skeys ? my_cnt[key] : ld_cg(a.cnt + (uint64_t) key * R + r);
			base = __shfl_sync(kFull, base, leader);
			if (key >= 0) {
				a.order[base + __popc(mm & lanemask_lt())] = (uint32_t) v;
				if (lane == leader) {
					if (skeys) my_cnt[key] = base + __popc(mm);
					else a.cnt[(uint64_t) key * R + r] = base + __popc(mm);
				}
			}
			__syncwarp();
		}
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t[1] = global_timer_ns();
	if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;

	// ---- 2. path counts, level by level ----------------------------------
	unsigned long long e_fwd = 0, e_rev = 0;
	bool pushed = false;      // the level before was pushed
	uint32_t pb = ld_cg(a.kstart);  // where the level before starts in `order`
	for (uint32_t d = 1; d <= depth; ++d) {
		const uint32_t bb = ld_cg(a.kstart + kBcClasses * d), be = ld_cg(a.kstart + kBcClasses * d + 1);
		// the counts of a pushed level are in lvx alone so far
		if (pushed)
			for (uint32_t i = pb + blockIdx.x * kBcThreads + threadIdx.x; i < bb; i += gridDim.x * kBcThreads) {
				const uint32_t v = ld_cg(a.order + i);
				a.sigma[v] = ld_cg(reinterpret_cast<const uint32_t *>(a.lvx + v) + 1);
			}
		// push where the level before has few vertices and less than half the
		// out-edges of this one's in-edges (the first levels, whose vertices
		// have the hubs' long in-edge lists: 94 us for the second level of a
		// Pokec-shape source whose first has two vertices)
		const uint32_t before = bb - pb;
		pushed = d < kBcTraceLevels && before <= kBcSmemBig &&
				2ull * ld_cg(&ctl->lv_deg[0][d - 1]) < ld_cg(&ctl->lv_deg[1][d]);
		if (pushed) {
			push_paths(a, pb, before, (int) d, use8, &e_fwd);
			pb = bb;
			if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;
			if (blockIdx.x == 0 && threadIdx.x == 0 && d < kBcTraceLevels) ctl->t_fwd[d] = global_timer_ns();
			continue;
		}
		pb = bb;
		const uint32_t nbig = be - bb;
		if (nbig > kBcSmemBig) {
			if (!big_chunks_global<true>(a, bb, nbig, (int) d - 1, use8, epoch)) return;
			if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;
			for (uint32_t i = gw; i < nbig; i += tw) {
				const uint32_t v = ld_cg(a.order + bb + i);
				const uint32_t s = big_finish_sum<true>(a, i, true);
				if (lane == 0) {
					finish_vertex<true>(a, v, s);
					e_fwd += a.in_off[v + 1] - a.in_off[v];
				}
			}
		}
		level_sums<true>(a, d, (int) d - 1, nbig <= kBcSmemBig, false, use8, &e_fwd);
		if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;
		if (blockIdx.x == 0 && threadIdx.x == 0 && d < kBcTraceLevels) ctl->t_fwd[d] = global_timer_ns();
	}
	if (pushed) {
		const uint32_t end = ld_cg(a.kstart + kBcClasses * (depth + 1));
		for (uint32_t i = pb + blockIdx.x * kBcThreads + threadIdx.x; i < end; i += gridDim.x * kBcThreads) {
			const uint32_t v = ld_cg(a.order + i);
			a.sigma[v] = ld_cg(reinterpret_cast<const uint32_t *>(a.lvx + v) + 1);
		}
		if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t[2] = global_timer_ns();

	// ---- 3. dependency sums, deepest level first ---------------------------
	for (int d = (int) depth; d >= 0; --d) {
		const bool deepest = (uint32_t) d == depth;
		const uint32_t bb = ld_cg(a.kstart + kBcClasses * d), be = ld_cg(a.kstart + kBcClasses * d + 1);
		const uint32_t me = ld_cg(a.kstart + kBcClasses * d + kBcClasses - 2);
		const uint32_t se = ld_cg(a.kstart + kBcClasses * d + kBcClasses);
		const uint32_t nbig = be - bb;
		if (!deepest && nbig > kBcSmemBig) {
			if (!big_chunks_global<false>(a, bb, nbig, d + 1, use8, epoch)) return;
			if (!grid_sync(ctl->bar, epoch, &ctl->err)) return;
			for (uint32_t i = gw; i < nbig; i += tw) {
				const uint32_t v = ld_cg(a.order + bb + i);
				const float s = big_finish_sum<false>(a, i, true);
				if (lane == 0) {
					finish_vertex<false>(a, v, s);
					e_rev += a.row_off[v + 1] - a.row_off[v];
				}
			}
		}
		level_sums<false>(a, (uint32_t) d, d + 1, nbig <= kBcSmemBig, deepest, use8, &e_rev);
		if (d > 0 && !grid_sync(ctl->bar, epoch, &ctl->err)) return;
		if (blockIdx.x == 0 && threadIdx.x == 0 && (uint32_t) d < kBcTraceLevels) {
			ctl->t_rev[d] = global_timer_ns();
			ctl->lv_vertices[d] = se - bb;
			ctl->lv_big[d] = be - bb;
			ctl->lv_medium[d] = me - be;
		}
	}
	{
		const unsigned long long ef = block_sum(e_fwd);
		const unsigned long long er = block_sum(e_rev);
		if (threadIdx.x == 0) {
			if (ef) atomicAdd(&ctl->edges_fwd, ef);
			if (er) atomicAdd(&ctl->edges_rev, er);
			ctl->depth = depth;
		}
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t[3] = global_timer_ns();
}

} // namespace

int bc_launch(const BcArgs &a, int num_sms, cudaStream_t st, int *grid) {
	int per_sm = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bc, kBcThreads, 0) != cudaSuccess || per_sm < 1)
		return BFS_ECUDA;
	per_sm = std::min(per_sm, 2);
	const int g = std::min<int>(num_sms * per_sm, (int) kBcMaxGrid);
	if (grid) *grid = g;
	if (cudaMemsetAsync(a.ctl, 0, sizeof(BcControl), st) != cudaSuccess) return BFS_ECUDA;
	BcArgs aa = a;
	void *args[] = {&aa};
	if (cudaLaunchCooperativeKernel((const void *) k_bc, dim3(g), dim3(kBcThreads), args, 0, st) != cudaSuccess)
		return BFS_ECUDA;
	return BFS_OK;
}

} // namespace bfsg
