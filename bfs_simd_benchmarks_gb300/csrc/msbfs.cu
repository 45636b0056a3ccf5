// msbfs.cu -- batched BFS: up to 4096 sources traversed together, bit-sliced.
//
// No counterpart in the reference, which runs one source per program run
// (apps/bfs_simd/bfs.cpp:1159); each source's levels equal what graph_prepare
// (apps/bfs_simd/bfs.cpp:753-963) computes for it.
//
// Layout (K = ceil(num_sources / 64) words, source i is bit i%64 of word i/64):
//   vis[v][K]          sources that have reached v
//   hist[p][v][K]      sources that reached v first at level base + p; the
//                      plane of level L is the frontier that level L expands
//   pmask[p][v]        bit k: word k of v's row in plane p is non-zero (the
//                      frontier's vertex set, and which words to read)
//   queue[L&1]         the frontier's vertices: degree <= kMsBig from the
//                      front, higher degree from the back
// A level is expanded either
//   - push (top-down) while the frontier holds few edges: a warp takes a
//     frontier vertex, loads its K words once and ORs the non-zero ones into
//     every out-neighbour's next words (64-bit atomics); a high-degree vertex
//     has its edges spread over every warp of the grid; or
//   - pull (bottom-up) once it holds many: destinations gather the words of
//     their frontier in-neighbours and stop as soon as every source that has a
//     frontier has reached them (per-destination early exit).  Up to
//     kMsRowWords words per vertex a lane (or 8 lanes) takes a destination and
//     reads whole rows; with more, a warp takes one and reads the non-zero
//     words it still lacks, in groups of 8, 16 or 32 lanes per row.  Destinations with many in-edges are cut into
//     chunks that warps all over the grid gather and OR together; the last one
//     finishes the destination, so that a pull level has one grid barrier.
//     (R-MAT scale 22, 4096 sources: the level with the most gathers 7.8 ->
//     4.8 ms; Pokec shape, 64 sources: 0.54 -> 0.26 ms.)
// Clearing, seeding, all levels and the edge count run in one cooperative
// launch, levels separated by a bounded-spin grid barrier; the output pass,
// its own launch, turns planes into uint8 levels [source][vertex] (255 =
// unreached) through a shared-memory transpose.  When a traversal is
// deeper than the planes allocated, the planes so far are written out, the
// current frontier plane becomes plane 0 and the traversal goes on; the later
// output passes merge into the bytes already written.
#include <algorithm>
#include <cstring>

#include "../../include/bfs_gb300.h"
#include "device_common.cuh"
#include "msbfs.h"

namespace bfsg {

constexpr int kMsThreads = 512;
constexpr int kMsWarps = kMsThreads / 32;
constexpr uint32_t kMsWq = 512;         // per-warp staged queue appends (pull)
// push: edges per lane and round trip (2^14 vertices, whose first frontier has a
// vertex of almost kMsBig edges: that level 38 -> 24 us)
constexpr int kMsPushEdges = 4;
constexpr uint32_t kMsBig = 1024;       // push: higher-degree vertices are spread over the grid
constexpr int kMsGather = 4;            // pull: frontier rows gathered per round
constexpr int kMsFinishRows = 2;        // push: touched rows finished per round
constexpr uint32_t kLaneMaxDeg = 32;    // pull, few words: destinations of at most this in-degree go one per lane
// Pull with more than kMsRowWords words: a block of 32 destinations is halved
// down to 4 while there are fewer than kMsBlocks per warp, and further while
// there are not blocks for half of the warps: a warp takes a block's destinations
// one after another (rmat, 16 edges a vertex: 2^12 vertices, 1,000 sources 549 ->
// 214 us; 2^14 546 -> 275; 2^16 543 -> 377; 2^18 1,142 -> 903).
constexpr uint32_t kMsBlocks = 4;
// Up to kMsRowWords words and this many words of state, one CTA per SM: a level
// is then a few chains of round trips and a grid barrier, which costs less among
// fewer CTAs (rmat, 16 edges a vertex, 60 sources: 2^14 vertices 177 -> 157 us,
// 2^16 162 -> 147, 2^17 206 -> 194; 2^18 264 -> 268).
// Up to kMsTinyState, a CTA on every other SM (2^14 vertices 155 -> 147 us, uniform
// 126 -> 115; 2^16 150 -> 163).
constexpr uint32_t kMsSmallState = 1u << 18, kMsTinyState = 1u << 15;
// Pull, few words: blocks taken at once (a power of two), as long as there are
// kMsClaims items per warp.  The counter gives out one claim in 0.8 ns, and where most
// destinations have no in-edges that is what a level waits for (uniform, 2^18 vertices
// of 16 edges, the first ids of 2^23: levels of 40 sources 1,014 -> 574 us, of 141 1,396
// -> 984; 2^20 of 8 in 2^25, 100 sources 6,950 -> 3,185; rmat, 2^23 vertices of 8 edges,
// 73 sources 2,340 -> 2,210).  With fewer items rmat 2^21 loses 2% and 2^22 4%.  More
// words per vertex lose by it at all sizes (2^23, 300 sources: 1,347 -> 2,041).
constexpr uint32_t kMsClaims = 12, kMsMaxClaim = 8;
constexpr uint32_t kMsRun = 8;          // pull, few words: chunks taken at once
constexpr uint32_t kMsMaxWords = 64;    // 4,096 sources
constexpr uint32_t kGroupMaxWords = 32; // pull: up to this many words, in-neighbour rows in lane groups
constexpr uint32_t kEmitW = 4;          // output tile: kV vertices x kW words (4: 256 sources), kV = threads / kW
constexpr uint32_t kEmitPlanes = 7;     // planes that a 3-bit index tells apart, with one value left for "none of them"
constexpr uint32_t kEmitUnits = 8;      // output tiles' words are split among CTAs below this many per CTA
// Words of a tile's shared memory per word of its vertices: 16 source quads, each
// a row of kV words with 4 more after every 16 (the second phase's 16-byte reads
// of 16 vertices per lane then fall on different banks), and the shift that puts
// the kW words of 32 / kW vertices on 32 different banks.
__host__ __device__ constexpr uint32_t emit_row(uint32_t kV) { return kV / 16 * 20; }
__host__ __device__ constexpr uint32_t emit_word_stride(uint32_t kV, uint32_t kW) { return 16 * emit_row(kV) + 32 / kW; }
// planes whose words are fetched a step ahead: two groups of seven; one where a
// vertex has more words, whose masks leave the second group nearly empty
__host__ __device__ constexpr uint32_t emit_slots(uint32_t kW) { return kW == 4 ? kEmitPlanes : 2 * kEmitPlanes; }
// shared bytes of an output tile: its quads' rows (or, in their place, its
// source rows); ahead: per thread a slot per plane of a step, and with kW = 4 its
// word masks
__host__ __device__ constexpr uint32_t emit_bytes(uint32_t kV, uint32_t kW, bool ahead) {
	return kW * emit_word_stride(kV, kW) * 4 + (ahead ? (emit_slots(kW) + (kW == 4 ? 4 : 0)) * kV * kW * 8 : 0);
}
constexpr uint32_t kMsRowWords = 4;     // pull: up to this many words per vertex, rows are read whole
constexpr uint32_t kEmitV = kMsThreads / kEmitW;  // the traversal kernel's tiles (its early output passes)
constexpr uint32_t kEmitBytes = emit_bytes(kEmitV, kEmitW, false);

__device__ __forceinline__ uint64_t ld_cg64(const uint64_t *p) { return __ldcg((const unsigned long long *) p); }
__device__ __forceinline__ uint64_t shfl64(uint64_t x, int src) {
	return (uint64_t) __shfl_sync(kFull, (unsigned long long) x, src);
}
__device__ __forceinline__ uint64_t shfl_xor64(uint64_t x, int mask) {
	return (uint64_t) __shfl_xor_sync(kFull, (unsigned long long) x, mask);
}
__device__ __forceinline__ uint32_t deg_of(const MsArgs &a, uint32_t v) {
	return __ldg(a.row_off + v + 1) - __ldg(a.row_off + v);
}

// Warp-aggregated append of the lanes with `small` / `big` set to the
// queue of the next level (small from the front, big from the back).
__device__ __forceinline__ void ms_append(const MsArgs &a, MsCounters *cn, uint32_t *qn, uint32_t v, bool small,
		bool big) {
	const unsigned ms = __ballot_sync(kFull, small);
	if (ms) {
		uint32_t base = 0;
		if (lane_id() == 0) base = atomicAdd(&cn->nact, (unsigned) __popc(ms));
		base = __shfl_sync(kFull, base, 0);
		if (small) qn[base + __popc(ms & lanemask_lt())] = v;
	}
	const unsigned mb = __ballot_sync(kFull, big);
	if (mb) {
		uint32_t base = 0;
		if (lane_id() == 0) base = atomicAdd(&cn->nbig, (unsigned) __popc(mb));
		base = __shfl_sync(kFull, base, 0);
		if (big) qn[a.n - 1 - (base + __popc(mb & lanemask_lt()))] = v;
	}
}

// Push: ORs u's non-zero frontier words into the next words of its out-edges
// [beg + first, end), taking 32 edges per warp step of `step`.  Warp-uniform.
__device__ __forceinline__ void ms_push_edges(const MsArgs &a, const uint64_t *cur, const uint64_t *actc,
		uint64_t *nxt, uint32_t u, uint32_t beg, uint32_t end) {
	const uint32_t K = a.K;
	const unsigned lane = lane_id();
	const uint64_t um = ld_cg64(actc + u);  // which of u's words are non-zero
	const uint32_t nz0 = (uint32_t) um, nz1 = (uint32_t) (um >> 32);
	const uint64_t w0 = (nz0 >> lane) & 1u ? ld_cg64(cur + (size_t) u * K + lane) : 0ull;
	const uint64_t w1 = (nz1 >> lane) & 1u ? ld_cg64(cur + (size_t) u * K + lane + 32) : 0ull;
	for (uint32_t i = 0; i < end - beg; i += 32 * kMsPushEdges) {
		uint32_t v[kMsPushEdges];
		bool ok[kMsPushEdges], fresh[kMsPushEdges];
#pragma unroll
		for (int j = 0; j < kMsPushEdges; ++j) {
			const uint32_t e = i + 32 * j + lane;
			ok[j] = e < end - beg;
			v[j] = ok[j] ? __ldg(a.col + beg + e) : 0u;
		}
#pragma unroll
		for (int j = 0; j < kMsPushEdges; ++j) fresh[j] = ok[j] && !ld_cg_u8(a.touched + v[j]);
		for (uint32_t m = nz0; m; m &= m - 1) {
			const int k = __ffs(m) - 1;
			const uint64_t w = shfl64(w0, k);
#pragma unroll
			for (int j = 0; j < kMsPushEdges; ++j)
				if (ok[j]) atomicOr((unsigned long long *) (nxt + (size_t) v[j] * K + k), (unsigned long long) w);
		}
		for (uint32_t m = nz1; m; m &= m - 1) {
			const int k = __ffs(m) - 1;
			const uint64_t w = shfl64(w1, k);
#pragma unroll
			for (int j = 0; j < kMsPushEdges; ++j)
				if (ok[j]) atomicOr((unsigned long long *) (nxt + (size_t) v[j] * K + k + 32), (unsigned long long) w);
		}
#pragma unroll
		for (int j = 0; j < kMsPushEdges; ++j)
			if (fresh[j]) a.touched[v[j]] = 1;
	}
}

// Push level, CTA 0: cuts the high-degree frontier vertices (the queue's back)
// into kMsPushChunk-edge chunks, listed in push_u / push_beg, so that warps
// all over the grid take them like small vertices.  A block-wide scan of the
// chunk counts, 512 vertices at a time.
__device__ void ms_push_chunk_list(const MsArgs &a, uint32_t lvl, uint32_t nb, uint32_t *scan_s) {
	const uint32_t *q = a.queue[lvl & 1];
	uint32_t running = 0;
	for (uint32_t base = 0; base < nb; base += blockDim.x) {
		const uint32_t i = base + threadIdx.x;
		uint32_t u = 0, c = 0, beg = 0, end = 0;
		if (i < nb) {
			u = ld_cg(q + a.n - 1 - i);
			beg = __ldg(a.row_off + u);
			end = __ldg(a.row_off + u + 1);
			c = (end - beg + kMsPushChunk - 1) / kMsPushChunk;
		}
		const uint32_t incl = warp_incl_scan(c);
		if (lane_id() == 31) scan_s[warp_id()] = incl;
		__syncthreads();
		uint32_t before = 0, total = 0;
		for (int w = 0; w < kMsWarps; ++w) {
			const uint32_t t = scan_s[w];
			if (w < (int) warp_id()) before += t;
			total += t;
		}
		uint32_t pos = running + before + incl - c;
		for (uint32_t k = 0; k < c && pos < a.push_cap; ++k, ++pos) {
			a.push_u[pos] = u;
			a.push_beg[pos] = beg + k * kMsPushChunk;
		}
		running += total;
		__syncthreads();
	}
	if (threadIdx.x == 0) a.ctl->push_chunks = min(running, a.push_cap);
}

// Push level with few edges: clears only the rows that will receive words (the
// first edge to reach one claims it in `touched`), instead of the whole plane.
// R-MAT scale 22 with 64 words per vertex: a plane is 2 GiB, 0.33 ms to clear;
// levels of up to n / kMsMarkDiv edges take 0.02 to 0.06 ms this way.
constexpr uint32_t kMsMarkDiv = 8;
constexpr uint32_t kMsMarkBig = 64;  // high-degree frontier vertices, one after the other by the whole grid
__device__ __forceinline__ void ms_mark_edges(const MsArgs &a, uint64_t *nxt, uint64_t e0, uint32_t end) {
	const unsigned lane = lane_id();
	const uint64_t e = e0 + lane;
	const uint32_t v = e < end ? __ldg(a.col + e) : 0u;
	bool mine = e < end && !ld_cg_u8(a.touched + v);
	if (mine) {
		const uint32_t bit = 1u << (8 * (v & 3u));
		mine = !(atomicOr(reinterpret_cast<unsigned *>(a.touched + (v & ~3u)), bit) & bit);
	}
	for (uint32_t m = __ballot_sync(kFull, mine); m; m &= m - 1) {
		uint64_t *row = nxt + (size_t) __shfl_sync(kFull, v, __ffs(m) - 1) * a.K;
		for (uint32_t k = lane; k < a.K; k += 32) row[k] = 0ull;
	}
}
__device__ void ms_push_mark(const MsArgs &a, uint32_t lvl, uint64_t *nxt, uint32_t nq, uint32_t nb) {
	const uint32_t *q = a.queue[lvl & 1];
	const uint32_t gwarp = blockIdx.x * kMsWarps + warp_id();
	const uint32_t nwarps = gridDim.x * kMsWarps;
	for (uint32_t i = gwarp; i < nq; i += nwarps) {
		const uint32_t u = ld_cg(q + i), end = __ldg(a.row_off + u + 1);
		for (uint64_t e = __ldg(a.row_off + u); e < end; e += 32) ms_mark_edges(a, nxt, e, end);
	}
	for (uint32_t i = 0; i < nb; ++i) {
		const uint32_t u = ld_cg(q + a.n - 1 - i), end = __ldg(a.row_off + u + 1);
		for (uint64_t e = (uint64_t) __ldg(a.row_off + u) + 32 * gwarp; e < end; e += 32 * nwarps) ms_mark_edges(a, nxt, e, end);
	}
}

__device__ void ms_push(const MsArgs &a, uint32_t lvl, const uint64_t *cur, const uint64_t *actc, uint64_t *nxt, uint32_t nq,
		uint32_t nb) {
	const uint32_t *q = a.queue[lvl & 1];
	const uint32_t gwarp = blockIdx.x * kMsWarps + warp_id();
	const uint32_t nwarps = gridDim.x * kMsWarps;
	for (uint32_t i = gwarp; i < nq; i += nwarps) {
		const uint32_t u = ld_cg(q + i);
		ms_push_edges(a, cur, actc, nxt, u, __ldg(a.row_off + u), __ldg(a.row_off + u + 1));
	}
	if (!nb) return;
	const uint32_t nc = ld_volatile(&a.ctl->push_chunks);
	for (uint32_t c = gwarp; c < nc; c += nwarps) {
		const uint32_t u = ld_cg(a.push_u + c), beg = ld_cg(a.push_beg + c);
		const uint32_t end = run_end(beg, kMsPushChunk, __ldg(a.row_off + u + 1));
		ms_push_edges(a, cur, actc, nxt, u, beg, end);
	}
}

// The next-frontier mask of a row whose new words lanes hold (word l, l + 32).
__device__ __forceinline__ uint64_t row_mask(uint64_t n0, uint64_t n1) {
	return (uint64_t) __ballot_sync(kFull, n0 != 0ull) | ((uint64_t) __ballot_sync(kFull, n1 != 0ull) << 32);
}

// After a push level: the OR'ed words lose the bits already visited, the rest
// are new, go into vis and put v into the next frontier.  A warp takes 32
// vertices, then works through the touched ones together (K words each).
__device__ void ms_push_finish(const MsArgs &a, uint32_t lvl, uint64_t *nxt, uint64_t *actn, unsigned long long &actdeg,
		unsigned long long *s_act) {
	const uint32_t K = a.K;
	const unsigned lane = lane_id();
	uint32_t *qn = a.queue[(lvl + 1) & 1];
	MsCounters *cn = &a.ctl->ctr[(lvl + 1) % 3];
	const uint32_t gwarp = blockIdx.x * kMsWarps + warp_id();
	const uint32_t nwarps = gridDim.x * kMsWarps;
	uint64_t newacc[2] = {0ull, 0ull};
	for (uint32_t vb = gwarp * 32; vb < a.n; vb += nwarps * 32) {
		const uint32_t v = vb + lane;
		const bool t = v < a.n && ld_cg_u8(a.touched + v);
		uint32_t anym = 0;
		for (uint32_t tm = __ballot_sync(kFull, t); tm;) {
			// kMsFinishRows touched rows at a time, the loads of all of them in flight
			size_t row[kMsFinishRows];
			uint32_t j[kMsFinishRows];
			uint64_t w[kMsFinishRows][2], vv[kMsFinishRows][2];
#pragma unroll
			for (int r = 0; r < kMsFinishRows; ++r) {
				j[r] = tm ? (uint32_t) __ffs(tm) - 1 : 32u;
				tm &= tm - 1;
				row[r] = (size_t) (vb + (j[r] & 31u)) * K;
#pragma unroll
				for (int h = 0; h < 2; ++h) {
					const uint32_t k = lane + 32 * h;
					const bool ld = j[r] < 32 && k < K;
					w[r][h] = ld ? ld_cg64(nxt + row[r] + k) : 0ull;
					vv[r][h] = ld ? ld_cg64(a.vis + row[r] + k) : 0ull;
				}
			}
#pragma unroll
			for (int r = 0; r < kMsFinishRows; ++r) {
				if (j[r] == 32u) break;
				uint64_t nw[2];
#pragma unroll
				for (int h = 0; h < 2; ++h) {
					const uint32_t k = lane + 32 * h;
					nw[h] = w[r][h] & ~vv[r][h];
					if (nw[h] != w[r][h]) nxt[row[r] + k] = nw[h];
					if (nw[h]) a.vis[row[r] + k] = vv[r][h] | nw[h];
					newacc[h] |= nw[h];
				}
				const uint64_t mask = row_mask(nw[0], nw[1]);
				if (lane == 0) actn[vb + j[r]] = mask;
				if (mask) anym |= 1u << j[r];
			}
		}
		if (t) a.touched[v] = 0;
		else if (v < a.n) actn[v] = 0;
		const bool any = (anym >> lane) & 1u;
		const uint32_t d = any ? deg_of(a, v) : 0u;
		ms_append(a, cn, qn, v, any && d <= kMsBig, any && d > kMsBig);
		actdeg += d;
	}
	if (lane < a.K && newacc[0]) atomicOr(s_act + lane, (unsigned long long) newacc[0]);
	if (lane + 32 < a.K && newacc[1]) atomicOr(s_act + lane + 32, (unsigned long long) newacc[1]);
}

// Pull appends: small vertices go through a per-warp shared buffer (one
// atomicAdd per kMsWq vertices), big ones straight to the queue's back.
__device__ __forceinline__ void ms_wq_flush(MsCounters *cn, uint32_t *qn, uint32_t *wbuf, uint32_t &wn) {
	__syncwarp();
	if (wn) {
		uint32_t base = 0;
		if (lane_id() == 0) base = atomicAdd(&cn->nact, wn);
		base = __shfl_sync(kFull, base, 0);
		for (uint32_t i = lane_id(); i < wn; i += 32) qn[base + i] = wbuf[i];
	}
	__syncwarp();
	wn = 0;
}

// The bits a complete word of lane's word (lane + 32 * h) holds.
struct FullMask {
	uint64_t f0, f1;
	// `act` (may be null: every source): the level's active words
	__device__ __forceinline__ FullMask(const MsArgs &a, unsigned lane, const unsigned long long *act = nullptr) {
		const uint64_t last = a.last_bits == 64 ? ~0ull : ((1ull << a.last_bits) - 1);
		f0 = lane < a.K ? (lane == a.K - 1 ? last : ~0ull) : 0ull;
		f1 = lane + 32 < a.K ? (lane + 32 == a.K - 1 ? last : ~0ull) : 0ull;
		if (act) {
			if (lane < a.K) f0 &= ld_cg64((const uint64_t *) act + lane);
			if (lane + 32 < a.K) f1 &= ld_cg64((const uint64_t *) act + lane + 32);
		}
	}
	__device__ __forceinline__ bool complete(uint64_t x0, uint64_t x1) const {
		return __all_sync(kFull, (x0 & f0) == f0 && (x1 & f1) == f1);
	}
};

// ORs into acc the frontier words of the in-neighbours in [beg, end) until
// every source has reached the destination.  Only words that are non-zero in
// the neighbour's row and still incomplete in the destination's are read.
// Returns true when it stopped early.  Warp-uniform.
__device__ __forceinline__ bool ms_gather(const MsArgs &a, const uint64_t *cur, const uint64_t *actc, uint32_t beg,
		uint32_t end, uint32_t u, uint64_t um, const FullMask &fm, uint64_t vis0, uint64_t vis1, uint64_t &acc0, uint64_t &acc1,
		unsigned long long &gathered) {
	const uint32_t K = a.K;
	const unsigned lane = lane_id();
	bool done = false;
	uint32_t loads = 0;
	for (uint32_t e0 = beg; e0 < end && !done; e0 += 32) {
		if (e0 != beg) um = e0 + lane < end ? ld_cg64(actc + u) : 0ull;
		const uint32_t en = e0 + 32 + lane, un = en < end ? __ldg(a.in_src + en) : 0u;
		uint32_t lm = __ballot_sync(kFull, um != 0ull);
		while (lm && !done) {
			const bool need0 = ((acc0 | vis0) & fm.f0) != fm.f0;
			const bool need1 = ((acc1 | vis1) & fm.f1) != fm.f1;
			uint64_t g0[kMsGather], g1[kMsGather];
#pragma unroll
			for (int t = 0; t < kMsGather; ++t) {
				uint32_t ut = 0;
				uint64_t mt = 0;
				if (lm) {
					const int src_lane = __ffs(lm) - 1;
					lm &= lm - 1;
					ut = __shfl_sync(kFull, u, src_lane);
					mt = shfl64(um, src_lane);
				}
				const uint64_t *r = cur + (size_t) ut * K;
				const bool l0 = need0 && ((mt >> lane) & 1ull), l1 = need1 && ((mt >> (lane + 32)) & 1ull);
				g0[t] = l0 ? ld_cg64(r + lane) : 0ull;
				g1[t] = l1 ? ld_cg64(r + lane + 32) : 0ull;
				loads += (uint32_t) l0 + (uint32_t) l1;  // words read by this lane
			}
#pragma unroll
			for (int t = 0; t < kMsGather; ++t) { acc0 |= g0[t]; acc1 |= g1[t]; }
			done = fm.complete(acc0 | vis0, acc1 | vis1);
		}
		u = un;
	}
	gathered += loads;
	return done;
}

__device__ __forceinline__ uint64_t warp_or64(uint64_t x) {
#pragma unroll
	for (int d = 16; d > 0; d >>= 1) x |= shfl_xor64(x, d);
	return x;
}

// ms_gather for kMsRowWords < K <= kGroupMaxWords words per vertex: the warp is
// split into groups of kLanes lanes (8, or 16 for more than 8 words); of g groups,
// each takes every g-th in-neighbour and reads its row (lane k its words k, and
// k + 16 of more than 16), so a round reads g kMsGather rows; the groups' words are
// OR-ed together after every round for the early exit.  `vis0` and `f0` are lane's
// word; so is the result.
// (Sharing the frontier's neighbours out evenly, by __fns, cost more than idle
// groups: uniform, 2^18 vertices, 2^22 edges, 300 sources: 1.13 against 0.80 ms.
// With a warp per row as above 32 words, rmat, 2^20 vertices, 2^24 edges, 1,024
// sources: 3.81 against 2.63 ms; 2,048 sources: 4.46 against 3.71.)
template <int KK>
__device__ __forceinline__ uint64_t ms_gather_grouped(const MsArgs &a, const uint64_t *cur, const uint64_t *actc,
		uint32_t beg, uint32_t end, uint32_t u, uint64_t um, uint64_t f0, uint64_t vis0, unsigned long long &gathered) {
	constexpr uint32_t kLanes = KK > 8 ? 16 : 8;
	constexpr int kWords = KK / (int) kLanes;
	const uint32_t K = a.K;
	const unsigned lane = lane_id();
	const uint32_t k = lane % kLanes;
	uint32_t loads = 0;
	uint64_t f[kWords], have[kWords];
	bool full = true;
#pragma unroll
	for (int j = 0; j < kWords; ++j) {
		f[j] = shfl64(f0, k + kLanes * j);  // zero beyond the last word
		have[j] = shfl64(vis0, k + kLanes * j);
		full &= (have[j] & f[j]) == f[j];
	}
	bool done = __all_sync(kFull, full);
	for (uint32_t e0 = beg; e0 < end && !done; e0 += 32) {
		if (e0 != beg) um = e0 + lane < end ? ld_cg64(actc + u) : 0ull;
		const uint32_t en = e0 + 32 + lane, un = en < end ? __ldg(a.in_src + en) : 0u;
		uint32_t lm = __ballot_sync(kFull, um != 0ull) & ((kLanes == 8 ? 0x11111111u : 0x55555555u) << (lane / kLanes));
		while (!done && __any_sync(kFull, lm)) {
			uint64_t gv[kMsGather][kWords];
#pragma unroll
			for (int t = 0; t < kMsGather; ++t) {
				const int src = __ffs(lm) - 1;
				const uint32_t ut = __shfl_sync(kFull, u, src & 31);
				const uint64_t mt = shfl64(um, src & 31);
#pragma unroll
				for (int j = 0; j < kWords; ++j) {
					const bool ld = lm && (have[j] & f[j]) != f[j] && ((mt >> (k + kLanes * j)) & 1ull);
					gv[t][j] = ld ? ld_cg64(cur + (size_t) ut * K + k + kLanes * j) : 0ull;
					loads += ld;
				}
				lm &= lm - 1;
			}
			full = true;
#pragma unroll
			for (int j = 0; j < kWords; ++j) {
#pragma unroll
				for (int t = 0; t < kMsGather; ++t) have[j] |= gv[t][j];
				for (uint32_t d = kLanes; d < 32; d <<= 1) have[j] |= shfl_xor64(have[j], d);
				full &= (have[j] & f[j]) == f[j];
			}
			done = __all_sync(kFull, full);
		}
		u = un;
	}
	gathered += loads;
	return kWords == 2 && lane >= kLanes ? have[kWords - 1] : lane < KK ? have[0] : 0ull;
}

// What a pull level works on.
struct MsPull {
	const uint64_t *cur, *actc;  // the frontier's plane and word masks
	uint64_t *nxt, *actn;        // the next level's
	const unsigned long long *act;  // sources with a frontier at this level (null: every source)
	MsCounters *cn;
	uint32_t *qn;                // the next level's queue
	// a destination without a new word: its row of nxt is not written.  Every
	// reader of the planes goes by the masks (more than kMsRowWords words per
	// vertex, and no later pass over the planes that reads them whole).
	bool masked;
};

// ---- pull with at most kMsRowWords words per vertex -----------------------
// A row is one sector at most, so a neighbour's row is read straight away
// (zero where it is not in the frontier) instead of its mask first and its
// words then: one round trip less per step.

template <int KK> __device__ __forceinline__ void row_ld(const uint64_t *p, uint64_t (&x)[KK]) {
	if constexpr (KK % 2 == 0) {
#pragma unroll
		for (int k = 0; k < KK; k += 2) {
			const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2 *>(p + k));
			x[k] = t.x;
			x[k + 1] = t.y;
		}
	} else {
#pragma unroll
		for (int k = 0; k < KK; ++k) x[k] = ld_cg64(p + k);
	}
}
// ORs the frontier rows of U in-neighbours into acc: the at, at + stride, ... -th of
// the `left` ones from in_src[e] on.
template <int KK, int U>
__device__ __forceinline__ uint32_t rows_or(const MsArgs &a, const uint64_t *cur, uint32_t e, uint32_t at, uint32_t stride,
		uint32_t left, uint64_t (&acc)[KK]) {
	uint32_t u[U], read = 0;
#pragma unroll
	for (int t = 0; t < U; ++t) u[t] = at + stride * t < left ? __ldg(a.in_src + e + at + stride * t) : 0xFFFFFFFFu;
	uint64_t x[U][KK];
#pragma unroll
	for (int t = 0; t < U; ++t) {
#pragma unroll
		for (int k = 0; k < KK; ++k) x[t][k] = 0ull;
		if (u[t] != 0xFFFFFFFFu) {
			row_ld<KK>(cur + (size_t) u[t] * KK, x[t]);
			read += KK;
		}
	}
#pragma unroll
	for (int t = 0; t < U; ++t)
#pragma unroll
		for (int k = 0; k < KK; ++k) acc[k] |= x[t][k];
	return read;
}
template <int KK>
__device__ __forceinline__ bool row_complete(const uint64_t (&x)[KK], const uint64_t (&y)[KK], const uint64_t (&f)[KK]) {
	bool r = true;
#pragma unroll
	for (int k = 0; k < KK; ++k) r &= ((x[k] | y[k]) & f[k]) == f[k];
	return r;
}

// The 32 destinations from vb (those of at most kMsPullBig in-edges): lanes
// walk the lists of up to kLaneMaxDeg in-edges, each its own, kRows rows per
// round trip; then groups of 8 lanes take the longer lists, four destinations
// at a time, 32 edges of each per round; a list's walk stops when every source
// that has a frontier has arrived.  All lanes then write their own destination.
template <int KK>
__device__ __forceinline__ void ms_pull_rows(const MsArgs &a, const MsPull &p, uint32_t vb, uint32_t nv, const uint64_t (&f)[KK],
		uint64_t (&newacc)[KK], unsigned long long &actdeg, unsigned long long &gathered, uint32_t *wbuf, uint32_t &wn) {
	constexpr int kRows = KK == 1 ? 8 : 4;
	const unsigned lane = lane_id();
	const uint32_t v = vb + lane;
	const bool valid = lane < nv;
	const uint32_t beg = valid ? __ldg(a.in_off + v) : 0u, end = valid ? __ldg(a.in_off + v + 1) : 0u;
	const bool small = valid && end - beg <= kMsPullBig;
	const bool needy = small && end > beg && !ld_cg_u8(a.done + v);
	uint64_t vis[KK], acc[KK];
#pragma unroll
	for (int k = 0; k < KK; ++k) vis[k] = acc[k] = 0ull;
	if (needy) row_ld<KK>(a.vis + (size_t) v * KK, vis);
	const bool open = needy && !row_complete(vis, acc, f);
	uint32_t read = 0;
	if (open && end - beg <= kLaneMaxDeg)
		for (uint32_t i = 0; i < end - beg && !row_complete(vis, acc, f); i += kRows)
			read += rows_or<KK, kRows>(a, p.cur, beg, i, 1, end - beg, acc);
	__syncwarp();
	for (uint32_t wm = __ballot_sync(kFull, open && end - beg > kLaneMaxDeg); wm;) {
		int j = -1;
		uint32_t m = wm;
#pragma unroll
		for (uint32_t g = 0; g < 4; ++g) {
			if (m && lane / 8 == g) j = __ffs(m) - 1;
			m &= m - 1u;
		}
		const uint32_t taken = wm & ~m;
		wm = m;
		const int src = j < 0 ? 0 : j;
		uint64_t gv[KK], ga[KK];
#pragma unroll
		for (int k = 0; k < KK; ++k) {
			gv[k] = shfl64(vis[k], src);
			ga[k] = 0ull;
		}
		uint32_t e = __shfl_sync(kFull, beg, src);
		uint32_t left = __shfl_sync(kFull, end, src) - e;
		for (bool go = j >= 0; __any_sync(kFull, go);) {
			if (go) read += rows_or<KK, 4>(a, p.cur, e, lane & 7u, 8, left, ga);
			e += 32;
			left -= min(left, 32u);
#pragma unroll
			for (int k = 0; k < KK; ++k)
#pragma unroll
				for (int d = 4; d > 0; d >>= 1) ga[k] |= shfl_xor64(ga[k], d);
			go = go && left && !row_complete(gv, ga, f);
		}
		// each destination's words from its group to its lane
		const int from = 8 * (__popc(taken & lanemask_lt()) & 3);
#pragma unroll
		for (int k = 0; k < KK; ++k) {
			const uint64_t x = shfl64(ga[k], from);
			if ((taken >> lane) & 1u) acc[k] = x;
		}
	}
	gathered += read;
	uint64_t mask = 0;
	if (small) {
		uint64_t w[KK];
#pragma unroll
		for (int k = 0; k < KK; ++k) {
			w[k] = acc[k] & ~vis[k] & f[k];
			newacc[k] |= w[k];
			if (w[k]) {
				mask |= 1ull << k;
				a.vis[(size_t) v * KK + k] = vis[k] | w[k];
			}
			p.nxt[(size_t) v * KK + k] = w[k];
		}
		p.actn[v] = mask;
		if (needy && row_complete(vis, w, f)) a.done[v] = 1;
	}
	const uint32_t d = mask ? deg_of(a, v) : 0u;
	actdeg += d;
	const uint32_t ms = __ballot_sync(kFull, mask && d <= kMsBig);
	if (wn + __popc(ms) > kMsWq) ms_wq_flush(p.cn, p.qn, wbuf, wn);
	if ((ms >> lane) & 1u) wbuf[wn + __popc(ms & lanemask_lt())] = v;
	wn += __popc(ms);
	if (mask && d > kMsBig) p.qn[a.n - 1 - atomicAdd(&p.cn->nbig, 1u)] = v;
}

// Chunks c0 .. c0 + cnt - 1 (at most 32 of them) of the destinations with more
// than kMsPullBig in-edges: lane t holds chunk c0 + t's facts; neighbouring
// chunks of one destination are read as one list and counted together, so that
// a destination costs one release of its words and not one per chunk (Pokec
// shape, 64 sources: 1.07 -> 0.88 ms; 11% of the warps' time was waiting for them).
template <int KK>
__device__ __forceinline__ void ms_pull_runs(const MsArgs &a, const MsPull &p, uint32_t c0, uint32_t cnt, const uint64_t (&f)[KK],
		uint64_t (&newacc)[KK], unsigned long long &actdeg, unsigned long long &gathered) {
	constexpr int kRows = KK == 1 ? 8 : 4;
	const unsigned lane = lane_id();
	const uint32_t c = c0 + min(lane, cnt - 1);
	const uint32_t v = __ldg(a.chunk_v + c), beg = __ldg(a.chunk_beg + c), slot = __ldg(a.chunk_slot + c);
	const uint32_t vbeg = __ldg(a.in_off + v), vend = __ldg(a.in_off + v + 1);
	uint64_t vis[KK];
	row_ld<KK>(a.vis + (size_t) v * KK, vis);
	const uint32_t openm = __ballot_sync(kFull, !row_complete(vis, vis, f));
	uint32_t read = 0;
	for (uint32_t t = 0; t < cnt;) {
		const uint32_t rv = __shfl_sync(kFull, v, t), rend = __shfl_sync(kFull, vend, t), rslot = __shfl_sync(kFull, slot, t);
		const uint32_t len = __popc(__ballot_sync(kFull, lane < cnt && v == rv));
		uint64_t acc[KK], have[KK];
#pragma unroll
		for (int k = 0; k < KK; ++k) {
			acc[k] = 0ull;
			have[k] = shfl64(vis[k], t);
		}
		uint64_t *bacc = a.big_acc + (size_t) rslot * KK;
		if ((openm >> t) & 1u) {
			uint32_t e = __shfl_sync(kFull, beg, t);
			uint32_t left = min(len * kMsChunk, rend - e);
			for (bool go = true; go && left; e += 32 * kRows, left -= min(left, 32u * kRows)) {
				read += rows_or<KK, kRows>(a, p.cur, e, lane, 32, left, acc);
				__syncwarp();
#pragma unroll
				for (int k = 0; k < KK; ++k) acc[k] = warp_or64(acc[k]);
				go = !row_complete(have, acc, f);
			}
#pragma unroll
			for (int k = 0; k < KK; ++k) {
				const uint64_t n = acc[k] & ~have[k] & f[k];
				if (lane == (unsigned) k && n) atomicOr((unsigned long long *) (bacc + k), (unsigned long long) n);
			}
		}
		__syncwarp();
		uint32_t before = 0;
		// releases this warp's words to, and acquires the other warps' from, those that count here
		if (lane == 0)
			asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(before) : "l"(a.big_cnt + rslot), "r"(len) : "memory");
		before = __shfl_sync(kFull, before, 0);
		if (before + len == (rend - __shfl_sync(kFull, vbeg, t) + kMsChunk - 1) / kMsChunk) {
			// every chunk is in: lane 0 finishes the destination
			if (lane == 0) {
				uint64_t mask = 0;
#pragma unroll
				for (int k = 0; k < KK; ++k) {
					const uint64_t n = ld_cg64(bacc + k);
					if (n) {
						bacc[k] = 0ull;
						a.vis[(size_t) rv * KK + k] = have[k] | n;
						newacc[k] |= n;
						mask |= 1ull << k;
					}
					p.nxt[(size_t) rv * KK + k] = n;
				}
				a.big_cnt[rslot] = 0u;
				p.actn[rv] = mask;
				if (mask) {
					const uint32_t d = deg_of(a, rv);
					actdeg += d;
					if (d > kMsBig) p.qn[a.n - 1 - atomicAdd(&p.cn->nbig, 1u)] = rv;
					else p.qn[atomicAdd(&p.cn->nact, 1u)] = rv;
				}
			}
			__syncwarp();
		}
		t += len;
	}
	gathered += read;
}

// ---- pull with more words per vertex --------------------------------------
// A warp screens 32 consecutive destinations at once (their in-edge ranges and
// "every source has arrived" flags, lane-parallel), then works through those
// with something to do one at a time: lane l owns words l and l + 32.
template <int KK>
__device__ __forceinline__ void ms_pull_words(const MsArgs &a, const MsPull &p, uint32_t vb, uint32_t nv, const FullMask &fm,
		uint64_t &new0, uint64_t &new1, unsigned long long &actdeg, unsigned long long &gathered, uint32_t *wbuf,
		uint32_t &wn) {
	const uint32_t K = a.K;
	const unsigned lane = lane_id();
	const bool w0 = lane < K, w1 = lane + 32 < K;
	const uint32_t vl = vb + lane;
	const bool valid = lane < nv;
	const uint32_t lbeg = valid ? __ldg(a.in_off + vl) : 0u, lend = valid ? __ldg(a.in_off + vl + 1) : 0u;
	const bool big = lend - lbeg > kMsPullBig;
	const bool needy = valid && !big && lend > lbeg && !ld_cg_u8(a.done + vl);
	const uint32_t needm = __ballot_sync(kFull, needy);
	if (valid && !needy && !big) p.actn[vl] = 0;
	if (!p.masked) {
		// rows of the block with nothing to do are zero
		const uint32_t bigm = __ballot_sync(kFull, big);
		uint64_t *blk = p.nxt + (size_t) vb * K;
		for (uint32_t x = lane; x < nv * K; x += 32)
			if (!(((needm | bigm) >> (x / K)) & 1u)) blk[x] = 0ull;
	}
	// a destination's first 32 in-neighbours are read, and its visited row is sent
	// for, while the one before it gathers (2^22 vertices, 4,096 sources: 24.6 -> 24.0 ms)
	const auto first_neighbours = [&](uint32_t m) {
		const int jj = __ffs(m) - 1;
		const uint32_t e = __shfl_sync(kFull, lbeg, jj) + lane;
		const uint64_t *r = a.vis + (size_t) (vb + jj) * K + 16 * lane;  // a line per lane
		if (16 * lane < K) asm volatile("prefetch.global.L2 [%0];" :: "l"(r));
		return e < __shfl_sync(kFull, lend, jj) ? __ldg(a.in_src + e) : 0u;
	};
	uint32_t un = needm ? first_neighbours(needm) : 0u;
	for (uint32_t m = needm; m; m &= m - 1) {
		const int jj = __ffs(m) - 1;
		const uint32_t v = vb + jj;
		const uint32_t beg = __shfl_sync(kFull, lbeg, jj), end = __shfl_sync(kFull, lend, jj);
		const size_t row = (size_t) v * K;
		const uint32_t u = un;
		const uint64_t um = beg + lane < end ? ld_cg64(p.actc + u) : 0ull;
		const uint64_t vis0 = w0 ? ld_cg64(a.vis + row + lane) : 0ull;
		const uint64_t vis1 = w1 ? ld_cg64(a.vis + row + lane + 32) : 0ull;
		if (m & (m - 1)) un = first_neighbours(m & (m - 1));
		uint64_t acc0 = 0, acc1 = 0;
		if constexpr (KK <= (int) kGroupMaxWords) {
			acc0 = ms_gather_grouped<KK>(a, p.cur, p.actc, beg, end, u, um, fm.f0, vis0, gathered);
		} else if (!fm.complete(vis0, vis1)) {
			ms_gather(a, p.cur, p.actc, beg, end, u, um, fm, vis0, vis1, acc0, acc1, gathered);
		}
		const uint64_t n0 = acc0 & ~vis0 & fm.f0, n1 = acc1 & ~vis1 & fm.f1;
		new0 |= n0;
		new1 |= n1;
		const uint64_t mask = row_mask(n0, n1);
		if (mask || !p.masked) {
			if (w0) p.nxt[row + lane] = n0;
			if (w1) p.nxt[row + lane + 32] = n1;
		}
		if (n0) a.vis[row + lane] = vis0 | n0;
		if (n1) a.vis[row + lane + 32] = vis1 | n1;
		const bool full = fm.complete(vis0 | n0, vis1 | n1);
		if (lane == 0) {
			p.actn[v] = mask;
			if (full) a.done[v] = 1;
		}
		if (mask) {
			const uint32_t d = deg_of(a, v);
			if (lane == 0) actdeg += d;
			if (d > kMsBig) {
				if (lane == 0) p.qn[a.n - 1 - atomicAdd(&p.cn->nbig, 1u)] = v;
			} else {
				if (lane == 0) wbuf[wn] = v;
				if (++wn == kMsWq) ms_wq_flush(p.cn, p.qn, wbuf, wn);
			}
		}
	}
}

// Chunk c of kMsChunk in-edges of a destination with more than kMsPullBig: the
// words it gathers are OR-ed into the destination's row of big_acc; the warp
// that completes the destination's last chunk writes its row, mask and queue
// entry and leaves its row of big_acc and its count at 0.
template <int KK>
__device__ __forceinline__ void ms_pull_chunk(const MsArgs &a, const MsPull &p, uint32_t c, const FullMask &fm,
		uint64_t &new0, uint64_t &new1, unsigned long long &actdeg, unsigned long long &gathered) {
	const uint32_t K = a.K;
	const unsigned lane = lane_id();
	const bool w0 = lane < K, w1 = lane + 32 < K;
	const uint32_t v = __ldg(a.chunk_v + c), beg = __ldg(a.chunk_beg + c), slot = __ldg(a.chunk_slot + c);
	const uint32_t vbeg = __ldg(a.in_off + v), vend = __ldg(a.in_off + v + 1);
	const uint32_t end = run_end(beg, kMsChunk, vend);
	const size_t row = (size_t) v * K;
	uint32_t u = 0;
	uint64_t um = 0;
	if (beg + lane < end) {
		u = __ldg(a.in_src + beg + lane);
		um = ld_cg64(p.actc + u);
	}
	const uint64_t vis0 = w0 ? ld_cg64(a.vis + row + lane) : 0ull;
	const uint64_t vis1 = w1 ? ld_cg64(a.vis + row + lane + 32) : 0ull;
	uint64_t *bacc = a.big_acc + (size_t) slot * K;
	if (!fm.complete(vis0, vis1)) {
		uint64_t acc0 = 0, acc1 = 0;
		if constexpr (KK <= (int) kGroupMaxWords) {
			acc0 = ms_gather_grouped<KK>(a, p.cur, p.actc, beg, end, u, um, fm.f0, vis0, gathered);
		} else {
			ms_gather(a, p.cur, p.actc, beg, end, u, um, fm, vis0, vis1, acc0, acc1, gathered);
		}
		const uint64_t n0 = acc0 & ~vis0 & fm.f0, n1 = acc1 & ~vis1 & fm.f1;
		if (n0) atomicOr((unsigned long long *) (bacc + lane), (unsigned long long) n0);
		if (n1) atomicOr((unsigned long long *) (bacc + lane + 32), (unsigned long long) n1);
	}
	__syncwarp();
	uint32_t before = 0;
	// releases this warp's words to, and acquires the other warps' from, those that count here
	if (lane == 0)
		asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(a.big_cnt + slot) : "memory");
	before = __shfl_sync(kFull, before, 0);
	if (before != (vend - vbeg + kMsChunk - 1) / kMsChunk - 1) return;
	__syncwarp();
	const uint64_t n0 = w0 ? ld_cg64(bacc + lane) : 0ull, n1 = w1 ? ld_cg64(bacc + lane + 32) : 0ull;
	if (n0) bacc[lane] = 0ull;
	if (n1) bacc[lane + 32] = 0ull;
	new0 |= n0;
	new1 |= n1;
	const uint64_t mask = row_mask(n0, n1);
	if (mask || !p.masked) {
		if (w0) p.nxt[row + lane] = n0;
		if (w1) p.nxt[row + lane + 32] = n1;
	}
	if (n0) a.vis[row + lane] = vis0 | n0;
	if (n1) a.vis[row + lane + 32] = vis1 | n1;
	if (lane == 0) {
		a.big_cnt[slot] = 0u;
		p.actn[v] = mask;
		if (mask) {
			const uint32_t d = deg_of(a, v);
			actdeg += d;
			if (d > kMsBig) p.qn[a.n - 1 - atomicAdd(&p.cn->nbig, 1u)] = v;
			else p.qn[atomicAdd(&p.cn->nact, 1u)] = v;
		}
	}
}

// The chunks from `item` on; returns the first item after them that this warp got.
template <int KK>
__device__ __forceinline__ uint32_t ms_pull_chunks(const MsArgs &a, const MsPull &p, uint32_t item, unsigned *counter,
		const FullMask &fm, unsigned long long &actdeg, unsigned long long &gathered, unsigned long long *s_act) {
	const unsigned lane = lane_id();
	uint64_t new0 = 0, new1 = 0;
	while (item < a.nchunks) {
		const uint32_t next = lane == 0 ? atomicAdd(counter, 1u) : 0u;
		ms_pull_chunk<KK>(a, p, item, fm, new0, new1, actdeg, gathered);
		item = __shfl_sync(kFull, next, 0);
	}
	if (new0) atomicOr(s_act + lane, (unsigned long long) new0);
	if (new1) atomicOr(s_act + lane + 32, (unsigned long long) new1);
	return item;
}

// The blocks of 32 destinations from `item` on.
template <int KK>
__device__ __forceinline__ void ms_pull_blocks(const MsArgs &a, const MsPull &p, uint32_t item, unsigned *counter,
		const FullMask &fm, unsigned long long &actdeg, unsigned long long &gathered, uint32_t *wbuf,
		unsigned long long *s_act) {
	const unsigned lane = lane_id();
	constexpr bool kRowWords = KK <= (int) kMsRowWords;
	constexpr int kN = kRowWords ? KK : 2;
	uint64_t f[kN], acc[kN];
#pragma unroll
	for (int k = 0; k < kN; ++k) {
		f[k] = kRowWords ? shfl64(fm.f0, k) : 0ull;
		acc[k] = 0ull;
	}
	uint32_t wn = 0;
	const uint32_t nruns = kRowWords ? a.nruns : a.nchunks;
	if constexpr (kRowWords) {
		while (item < nruns) {
			const uint32_t next = lane == 0 ? atomicAdd(counter, 1u) : 0u;
			const uint32_t c0 = item * a.run;
			ms_pull_runs<KK>(a, p, c0, min(a.run, a.nchunks - c0), f, acc, actdeg, gathered);
			item = gridDim.x * kMsWarps + __shfl_sync(kFull, next, 0);
		}
	}
	while (item < nruns + a.nclaims) {
		const uint32_t next = lane == 0 ? atomicAdd(counter, 1u) : 0u;
		if constexpr (kRowWords) {
			uint32_t vb = (item - nruns) * a.claim;  // (a.claim destinations, a power of two)
			do {
				ms_pull_rows<KK>(a, p, vb, min(32u, a.n - vb), f, acc, actdeg, gathered, wbuf, wn);
				vb += 32;
			} while ((vb & (a.claim - 1)) && vb < a.n);
		} else {
			const uint32_t vb = (item - nruns) << a.blk_shift;
			ms_pull_words<KK>(a, p, vb, min(1u << a.blk_shift, a.n - vb), fm, acc[0], acc[1], actdeg, gathered, wbuf, wn);
		}
		item = (kRowWords ? gridDim.x * kMsWarps : 0u) + __shfl_sync(kFull, next, 0);
	}
	ms_wq_flush(p.cn, p.qn, wbuf, wn);
	if constexpr (kRowWords) {
#pragma unroll
		for (int k = 0; k < KK; ++k) {
			const uint64_t x = warp_or64(acc[k]);
			if (lane == 0 && x) atomicOr(s_act + k, (unsigned long long) x);
		}
	} else {
		if (acc[0]) atomicOr(s_act + lane, (unsigned long long) acc[0]);
		if (acc[1]) atomicOr(s_act + lane + 32, (unsigned long long) acc[1]);
	}
}

// A pull level: the chunks of the many-in-edge destinations, then the blocks of
// destinations, handed to the warps one at a time, so that no barrier is needed
// between them: through a counter, the next one claimed while one runs; with few
// words a warp's first by its number (with more, that was 10% slower on 4,096
// sources).  The frontier's vertices are staged per warp:
// one atomic on the queue's length per kMsWq of them and not per block (together
// 2^18 vertices, 64 sources: 282 -> 270 us; 2^20 604 -> 586).  Two or more blocks
// at a time cost more in balance than they save on graphs of this size (2^20: 618).
template <int KK>
__device__ __forceinline__ void ms_pull(const MsArgs &a, const MsPull &p, unsigned *counter, unsigned long long &actdeg_out,
		unsigned long long &gathered_out, uint32_t *wq_base, unsigned long long *s_act) {
	const unsigned lane = lane_id();
	const FullMask fm(a, lane, p.act);
	unsigned long long actdeg = 0, gathered = 0;
	uint32_t item = warp_id() * gridDim.x + blockIdx.x;
	if constexpr (KK > (int) kMsRowWords) {
		item = __shfl_sync(kFull, lane == 0 ? atomicAdd(counter, 1u) : 0u, 0);
		if (item < a.nchunks) item = ms_pull_chunks<KK>(a, p, item, counter, fm, actdeg, gathered, s_act);
	}
	uint32_t *wbuf = wq_base + warp_id() * kMsWq;
	ms_pull_blocks<KK>(a, p, item, counter, fm, actdeg, gathered, wbuf, s_act);
	actdeg_out += actdeg;
	gathered_out += gathered;
}

// Planes [first, last] (levels base + p) -> uint8 levels [source][vertex].
// A CTA of 512 threads takes tiles of 128 vertices x 4 words (256 sources).
// 1. thread (vertex, word) -- the words of a vertex on neighbouring lanes, so
//    that a warp's load touches one sector per vertex -- builds the 64 level
//    bytes of its word's sources in 16 registers.  For every plane whose word
//    mask says the word is non-zero it loads the word.  Of 7 planes, a source's
//    bit is set in one at most: three words hold that plane's number in binary
//    (7: none), their bits are brought together as one nibble per source, and a
//    byte permute looks four nibbles up in the 8 bytes {lvl .. lvl + 6, 255} at
//    once.  That is about 100 instructions per 7 planes whatever they hold; an
//    XOR of looked-up byte masks per plane took 80 for each of them, the output
//    was bound by it (rmat, 2^20 vertices, 1,024 sources: 0.74 ms, 57% of the
//    issue slots, 58% of L1; now 0.40) and each lane of a warp read another
//    sector.  The 16 registers go to shared memory as [word][source quad][vertex].
// 2. thread (word, source quad, 16 vertices) reads its 16 words with 16-byte
//    loads, transposes them 4 x 4 bytes at a time (byte permutes) into the
//    16-byte pieces of its 4 source rows and stores those.
// `merge` combines with the bytes already in `levels` (a later segment of a
// traversal deeper than the planes) by a byte-wise minimum: every byte is
// below 255 in at most one segment.
// Source j of quad q (j < 4, q < 16) among its word's 64.
__device__ __forceinline__ constexpr uint32_t emit_source(uint32_t q, uint32_t j) { return q / 4 * 16 + q % 4 + 4 * j; }

// The 64 level bytes of a word's sources, lvl + t where plane w[t] has the
// source's bit and 255 where none has, combined into o (a source's bit is set
// in one plane at most, and 255 is all ones: an AND).
__device__ __forceinline__ void emit_bytes_of(const uint64_t (&w)[kEmitPlanes], uint32_t lvl, uint32_t (&o)[16]) {
	const uint32_t lo = lvl * 0x01010101u + 0x03020100u, hi = (lvl * 0x00010101u + 0x00060504u) | 0xFF000000u;
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		uint32_t x[kEmitPlanes];
#pragma unroll
		for (uint32_t t = 0; t < kEmitPlanes; ++t) x[t] = (uint32_t) (w[t] >> (32 * h));
		const uint32_t none = ~(x[0] | x[1] | x[2] | x[3] | x[4] | x[5] | x[6]);
		const uint32_t b0 = x[1] | x[3] | x[5] | none, b1 = x[2] | x[3] | x[6] | none, b2 = x[4] | x[5] | x[6] | none;
#pragma unroll
		for (uint32_t r = 0; r < 4; ++r) {  // nibble i of sel: the index of source 32 h + 4 i + r
			const uint32_t c1 = r ? b1 >> (r - 1) : b1 << 1, c2 = r < 2 ? b2 << (2 - r) : b2 >> (r - 2);
			const uint32_t sel = ((b0 >> r) & 0x11111111u) | (c1 & 0x22222222u) | (c2 & 0x44444444u);
			o[8 * h + r] &= __byte_perm(lo, hi, sel);
			o[8 * h + 4 + r] &= __byte_perm(lo, hi, sel >> 16);
		}
	}
}

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// kAhead (the launch of its own after the traversal): a step's words are copied
// to shared memory while the step before is looked up, transposed and stored;
// every thread copies what it reads itself, so that no barrier is between.  A
// CTA goes through a tile's words before it takes another tile, so that a
// tile's masks come from L1 and the neighbouring sectors of its rows from L2.
// Without kAhead (inside the traversal kernel) everything is read around L1.
//
// kShift: rows that do not start on 16-byte boundaries (n or `levels` not a
// multiple of 16).  Phase 2 then leaves its bytes in shared memory, row by row,
// and a third phase writes every row in 16-byte pieces of its own alignment,
// each put together from five words by funnel shifts; only the up to 15 bytes
// at either end of a tile's row go out in smaller stores.  (Straight from phase
// 2, a row on an odd address went out a byte at a time: Pokec shape, 64
// sources, 0.23 ms.)
__host__ __device__ constexpr uint32_t emit_row_bytes(uint32_t kV) { return kV + 16; }

// 4 bytes at any byte offset of shared memory
__device__ __forceinline__ uint32_t smem_u32(const uint8_t *p, uint32_t o) {
	const uint32_t *w = reinterpret_cast<const uint32_t *>(p + (o & ~3u));
	return __funnelshift_r(w[0], w[1], 8 * (o & 3u));
}
// The row's bytes [0, nv) at src -> dst: piece 0 up to dst's first 16-byte
// boundary, piece i the 16 bytes from the i-th one on.
__device__ __forceinline__ void emit_shifted(const uint8_t *src, uint8_t *dst, uint32_t nv, uint32_t piece, bool merge) {
	const uint32_t head = min(nv, (uint32_t) (-(uintptr_t) dst & 15u));
	uint32_t o = piece ? head + 16 * (piece - 1) : 0u;
	if (o >= nv) return;
	const uint32_t len = piece ? min(16u, nv - o) : head;
	if (len == 16) {
		const uint32_t *w = reinterpret_cast<const uint32_t *>(src + (o & ~3u));
		const uint32_t sh = 8 * (o & 3u);
		uint32_t x[5];
#pragma unroll
		for (int q = 0; q < 5; ++q) x[q] = w[q];
		uint4 y = make_uint4(__funnelshift_r(x[0], x[1], sh), __funnelshift_r(x[1], x[2], sh),
				__funnelshift_r(x[2], x[3], sh), __funnelshift_r(x[3], x[4], sh));
		if (merge) {
			const uint4 old = __ldcg(reinterpret_cast<const uint4 *>(dst + o));
			y = make_uint4(__vminu4(y.x, old.x), __vminu4(y.y, old.y), __vminu4(y.z, old.z), __vminu4(y.w, old.w));
		}
		*reinterpret_cast<uint4 *>(dst + o) = y;
		return;
	}
	if (merge) {
		for (uint32_t i = o; i < o + len; ++i) dst[i] = min(src[i], ld_cg_u8(dst + i));
		return;
	}
	// a head grows to the 16-byte boundary, a tail shrinks from it
	if (piece == 0 && head == nv && ((uintptr_t) (dst + nv) & 15u)) {  // both ends inside one piece
		for (; o < nv; ++o) dst[o] = src[o];
		return;
	}
	for (uint32_t b = piece ? 8u : 1u; b && b <= 8u; b = piece ? b / 2 : b * 2) {
		if (!(len & b)) continue;
		if (b == 1) dst[o] = src[o];
		else if (b == 2) *reinterpret_cast<uint16_t *>(dst + o) = (uint16_t) smem_u32(src, o);
		else if (b == 4) *reinterpret_cast<uint32_t *>(dst + o) = smem_u32(src, o);
		else *reinterpret_cast<uint2 *>(dst + o) = make_uint2(smem_u32(src, o), smem_u32(src, o + 4));
		o += b;
	}
}

template <bool kAhead, uint32_t kV, uint32_t kW, bool kShift>
__device__ __noinline__ void ms_emit(const MsArgs &a, uint8_t *levels, uint32_t ns, uint32_t base, uint32_t first, uint32_t last,
		bool merge, uint8_t *lev) {
	static_assert(!kShift || kW * 64 * emit_row_bytes(kV) <= kW * emit_word_stride(kV, kW) * 4, "source rows fit in the quads' place");
	constexpr uint32_t kThreads = kV * kW, kRow = emit_row(kV), kSlots = emit_slots(kW), kWordStride = emit_word_stride(kV, kW), kRows = kW * 64;
	const uint32_t K = a.K, n = a.n;
	const uint32_t vtiles = (n + kV - 1) / kV, wtiles = (K + kW - 1) / kW;
	const uint32_t vi = threadIdx.x / kW, wi = threadIdx.x % kW;
	const size_t pstride = (size_t) n * K;
	uint32_t *const sw = reinterpret_cast<uint32_t *>(lev);  // [wi][quad][kRow]
	uint8_t *const rows = lev;  // kShift: then [source][emit_row_bytes]
	// this thread's words of one step, a slot per plane (kAhead)
	uint64_t *const slot = reinterpret_cast<uint64_t *>(lev + kW * kWordStride * 4) + threadIdx.x;
	uint2 *const group = reinterpret_cast<uint2 *>(slot + kSlots * kThreads);
	// phase 2's item: rows of source quad rq (word rq / 16), vertices 16 cc ...
	const uint32_t rq = threadIdx.x / (kV / 16), cc = threadIdx.x % (kV / 16);
	const uint32_t rw = rq / 16, q2 = rq % 16;
	// a CTA takes a tile's words one after another, as many as leave every CTA work
	uint32_t len = wtiles;
	while (len > 1 && (uint64_t) vtiles * ((wtiles + len - 1) / len) < (uint64_t) kEmitUnits * gridDim.x) len = (len + 1) / 2;
	const uint32_t units = vtiles * ((wtiles + len - 1) / len);
	uint32_t unit = blockIdx.x, v0 = 0, kt = 0, kend = 0, l = first;
	const auto place = [&] {  // the unit's first tile
		v0 = unit % vtiles * kV;
		kt = unit / vtiles * len;
		kend = min(kt + len, wtiles);
	};
	// which of the step's planes have a non-zero word for this thread
	const auto step_planes = [&] { return min(last + 1 - l, 2 * kEmitPlanes); };
	const auto inside = [&] { return v0 + vi < n && kt * kW + wi < K; };
	const auto nonzero = [&] {
		if (!inside()) return 0u;
		const uint32_t cnt = step_planes(), k = kt * kW + wi;
		if (K <= kMsRowWords) return (1u << cnt) - 1u;  // rows of so few words are zero where nothing is
		if constexpr (kAhead) {
			const uint2 g[4] = {group[0], group[kThreads], group[2 * kThreads], group[3 * kThreads]};
			uint32_t nz = 0;
#pragma unroll
			for (int i = 0; i < 4; ++i) nz |= ((kt < 8 ? g[i].x : g[i].y) >> (4 * (kt % 8)) & 15u) << (4 * i);
			return nz;
		}
		uint32_t nz = 0;
		for (uint32_t t = 0; t < cnt; ++t) nz |= (uint32_t) (ld_cg64(a.pmask + (size_t) (l + t) * n + v0 + vi) >> k & 1u) << t;
		return nz;
	};
	// kAhead: the bits of this thread's words (every kW-th) in the step's masks, nibble kt of group i planes 4 i ..
	const auto masks = [&] {
		if (K <= kMsRowWords || !inside()) return;
		const uint32_t cnt = step_planes();
		const unsigned long long *pm = reinterpret_cast<const unsigned long long *>(a.pmask) + (size_t) l * n + v0 + vi;
#pragma unroll
		for (uint32_t i = 0; i < 4; ++i) {
			unsigned long long g = 0;
#pragma unroll
			for (uint32_t t = 4 * i; t < min(4 * i + 4, 2 * kEmitPlanes); ++t)
				if (t < cnt) g |= (__ldg(pm + (size_t) t * n) >> wi & 0x1111111111111111ull) << (t % 4);
			group[i * kThreads] = make_uint2((uint32_t) g, (uint32_t) (g >> 32));
		}
	};
	const auto plane_words = [&] { return a.hist + (size_t) l * pstride + (size_t) (v0 + vi) * K + kt * kW + wi; };
	const auto fetch = [&] {  // kAhead: the step's words -> the slots, asynchronously
		const uint32_t nz = nonzero();
		const uint64_t *pw = plane_words();
#pragma unroll
		for (uint32_t h = 0; h < kSlots / kEmitPlanes; ++h) {
			if (!(nz >> (h * kEmitPlanes))) break;
#pragma unroll
			for (uint32_t t = h * kEmitPlanes; t < (h + 1) * kEmitPlanes; ++t)
				if ((nz >> t) & 1u) cp_async8(slot + t * kThreads, pw + (size_t) t * pstride);
		}
		return nz;
	};
	if (unit >= units) return;
	place();
	if (kAhead) masks();
	uint32_t nz = kAhead ? fetch() : 0u;
	uint32_t o[16];
#pragma unroll
	for (int q = 0; q < 16; ++q) o[q] = 0xFFFFFFFFu;
	for (;;) {
		// 1. this thread's 64 level bytes, 14 planes a step
		if (!kAhead) nz = nonzero();
		else cp_async_wait();
#pragma unroll
		for (uint32_t h = 0; h < 2; ++h) {
			if (!(nz >> (h * kEmitPlanes))) break;
			const uint64_t *pw = plane_words();
			uint64_t w[kEmitPlanes];
#pragma unroll
			for (uint32_t t = 0; t < kEmitPlanes; ++t) {
				const uint32_t p = h * kEmitPlanes + t;
				w[t] = !((nz >> p) & 1u) ? 0ull : kAhead && p < kSlots ? slot[p * kThreads] : ld_cg64(pw + (size_t) p * pstride);
			}
			emit_bytes_of(w, base + l + h * kEmitPlanes, o);
		}
		const uint32_t tv0 = v0, k0 = kt * kW;
		const bool out = l + 2 * kEmitPlanes > last;
		bool more = true;
		l += 2 * kEmitPlanes;
		if (out) {
			l = first;
			if (++kt == kend) {
				unit += gridDim.x;
				more = unit < units;
				if (more) place();
			}
		}
		if (kAhead && more && (!out || kt == unit / vtiles * len || last - first >= 2 * kEmitPlanes)) masks();
		if (kAhead) nz = more ? fetch() : 0u;
		if (!out) continue;
		const uint32_t nv = min(kV, n - tv0), nrows = min(kRows, ns - k0 * 64);
		uint32_t *col = sw + wi * kWordStride + vi + vi / 16 * 4;
#pragma unroll
		for (int q = 0; q < 16; ++q) {
			col[q * kRow] = o[q];
			o[q] = 0xFFFFFFFFu;
		}
		__syncthreads();
		// 2. rows out: 16 vertices x 4 source rows per thread
		const uint32_t c = cc * 16, r0 = rw * 64 + emit_source(q2, 0);
		const bool piece = k0 + rw < K && r0 < nrows && c < nv;
		uint32_t y[4][4];  // y[b][g]: source r0 + 4 b, vertices c + 4g .. c + 4g + 3
		if (piece) {
			const uint4 *sp = reinterpret_cast<const uint4 *>(sw + rw * kWordStride + q2 * kRow + cc * 20);
			uint32_t x[16];
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				const uint4 u = sp[j];
				x[4 * j] = u.x;
				x[4 * j + 1] = u.y;
				x[4 * j + 2] = u.z;
				x[4 * j + 3] = u.w;
			}
#pragma unroll
			for (int g = 0; g < 4; ++g) {
				const uint32_t t0 = __byte_perm(x[4 * g], x[4 * g + 1], 0x5140);
				const uint32_t t1 = __byte_perm(x[4 * g + 2], x[4 * g + 3], 0x5140);
				const uint32_t t2 = __byte_perm(x[4 * g], x[4 * g + 1], 0x7362);
				const uint32_t t3 = __byte_perm(x[4 * g + 2], x[4 * g + 3], 0x7362);
				y[0][g] = __byte_perm(t0, t1, 0x5410);
				y[1][g] = __byte_perm(t0, t1, 0x7632);
				y[2][g] = __byte_perm(t2, t3, 0x5410);
				y[3][g] = __byte_perm(t2, t3, 0x7632);
			}
		}
		if (kShift) __syncthreads();  // the source rows take the quads' place
		if (piece) {
#pragma unroll
			for (int b = 0; b < 4; ++b) {
				if constexpr (kShift) {
					*reinterpret_cast<uint4 *>(rows + (r0 + 4 * b) * emit_row_bytes(kV) + c) =
							make_uint4(y[b][0], y[b][1], y[b][2], y[b][3]);
					continue;
				}
				if (r0 + 4 * b >= nrows) break;
				// whole pieces of aligned rows
				uint4 *const d = reinterpret_cast<uint4 *>(levels + (size_t) (k0 * 64 + r0 + 4 * b) * n + tv0 + c);
				uint4 z = make_uint4(y[b][0], y[b][1], y[b][2], y[b][3]);
				if (merge) {
					const uint4 old = __ldcg(d);
					z = make_uint4(__vminu4(z.x, old.x), __vminu4(z.y, old.y), __vminu4(z.z, old.z), __vminu4(z.w, old.w));
				}
				*d = z;
			}
		}
		if (kShift) {
			__syncthreads();
			constexpr uint32_t kPieces = kV / 16 + 1;
			for (uint32_t i = threadIdx.x; i < nrows * kPieces; i += blockDim.x) {
				const uint32_t r = i / kPieces;
				emit_shifted(rows + r * emit_row_bytes(kV), levels + (size_t) (k0 * 64 + r) * n + tv0, nv, i % kPieces, merge);
			}
		}
		if (!more) return;
		__syncthreads();
	}
}

// An early output pass: the planes base .. lvl go out, lvl's becomes plane 0.  Two
// grid barriers after `epoch`; false where one gave up.  (A function: inside the
// traversal kernel, its loops and calls cost the pulls registers: levels of 200 sources,
// rmat, 2^20 vertices, 1,015 -> 930 us, of 141 885 -> 838; of 73, on a small unpermuted
// graph, 345 -> 352.)
__device__ __noinline__ bool ms_spill(const MsArgs &a, uint8_t *levels, uint32_t ns, uint32_t base, uint32_t lvl, uint8_t *lev,
		unsigned epoch) {
	const uint32_t stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
	const size_t nK = (size_t) a.n * a.K;
	const uint32_t first = base == 0 ? 0 : 1;
	// rows that all start on 16 bytes need no shifting: the level with the pass, 60 sources,
	// uniform, 2^21 vertices, 650 -> 591 us
	if (a.n % 16 == 0 && (uintptr_t) levels % 16 == 0)
		ms_emit<false, kEmitV, kEmitW, false>(a, levels, ns, base, first, lvl - base, base != 0, lev);
	else ms_emit<false, kEmitV, kEmitW, true>(a, levels, ns, base, first, lvl - base, base != 0, lev);
	if (!grid_sync(a.ctl->bar, epoch, &a.ctl->err, a.wait_limit_ns, a.hold_barrier)) return false;
	const uint64_t *src = a.hist + (size_t) (lvl - base) * nK;
	for (size_t i = t0; i < nK; i += stride) a.hist[i] = ld_cg64(src + i);
	const uint64_t *msrc = a.pmask + (size_t) (lvl - base) * a.n;
	for (uint32_t i = t0; i < a.n; i += stride) a.pmask[i] = ld_cg64(msrc + i);
	return grid_sync(a.ctl->bar, epoch, &a.ctl->err, a.wait_limit_ns, a.hold_barrier);
}

// KK: words per vertex up to kMsRowWords; for more, 8, 16, 32 (kGroupMaxWords) or 64
// (kMsMaxWords) for up to as many: one kernel each, so that only one form of the pull shares
// the registers and its arguments are read where they lie (as calls of one
// kernel, with arguments by reference, the pulls' accesses to local memory were
// a third of their L1 traffic: 2^22 vertices, 4,096 sources, 28.6 against 24.6 ms).
template <int KK>
__global__ void __launch_bounds__(kMsThreads, 2) k_ms_bfs(const __grid_constant__ MsArgs a, const uint32_t *sources, uint32_t ns,
		uint8_t *levels) {
	__shared__ unsigned long long red[kMsWarps];
	// an early output pass's tile; while levels run, the warps' staged appends
	__shared__ __align__(16) uint8_t lev[kEmitBytes];
	static_assert(kMsWarps * kMsWq * 4 <= kEmitBytes, "the appends fit in the tile");
	uint32_t *const wq = reinterpret_cast<uint32_t *>(lev);
	MsControl *ctl = a.ctl;
	const uint32_t stride = gridDim.x * blockDim.x;
	const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
	const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
	const size_t nK = (size_t) a.n * a.K;
	unsigned epoch = 0;  // grid barriers passed (the control block, and its arrival count, start zeroed)
	if (leader) ctl->stats.t_start = global_timer_ns();
	// clear (the control block was zeroed by the host)
	for (size_t i = t0; i < nK; i += stride) { a.vis[i] = 0; a.hist[i] = 0; }
	for (size_t i = t0; i < (size_t) a.nbig_in * a.K; i += stride) a.big_acc[i] = 0;
	for (uint32_t i = t0; i < a.nbig_in; i += stride) a.big_cnt[i] = 0;
	for (uint32_t i = t0; i < a.n; i += stride) {
		a.pmask[i] = 0;
		a.done[i] = 0;
		a.touched[i] = 0;
		a.seed_flag[i] = 0;
	}
	bool ok = grid_sync(ctl->bar, epoch, &ctl->err, a.wait_limit_ns, a.hold_barrier);
	// plane 0: every source reaches itself
	if (ok) {
		for (uint32_t i = t0; i < ns; i += stride) {
			const uint32_t v = sources[i];
			if (v >= a.n) {  // device-resident sources are checked here
				atomicExch(&ctl->err, BFS_EARG);
				continue;
			}
			const size_t x = (size_t) v * a.K + i / 64;
			const unsigned long long bit = 1ull << (i % 64);
			atomicOr((unsigned long long *) (a.hist + x), bit);
			atomicOr((unsigned long long *) (a.vis + x), bit);
			atomicOr((unsigned long long *) (a.pmask + v), 1ull << (i / 64));
			if (atomicExch(a.seed_flag + v, 1u) == 0u) {
				const uint32_t d = deg_of(a, v);
				if (d > kMsBig) a.queue[0][a.n - 1 - atomicAdd(&ctl->ctr[0].nbig, 1u)] = v;
				else a.queue[0][atomicAdd(&ctl->ctr[0].nact, 1u)] = v;
				atomicAdd(&ctl->ctr[0].act_deg, (unsigned long long) d);
			}
		}
		ok = grid_sync(ctl->bar, epoch, &ctl->err, a.wait_limit_ns, a.hold_barrier);
	}
	if (leader) ctl->stats.t_levels0 = global_timer_ns();
	unsigned long long gathered = 0;
	uint32_t base = 0, lvl = 0;
	bool complete = false;
	__shared__ unsigned long long s_act[64];  // this CTA's OR of the next frontier's words
	for (; ok; ++lvl) {
		MsCounters *cc = &ctl->ctr[lvl % 3];
		const uint32_t nq = ld_volatile(&cc->nact), nb = ld_volatile(&cc->nbig);
		const unsigned long long qdeg = ld_volatile_u64(&cc->act_deg);
		if (nq + nb == 0) { complete = true; break; }
		if (lvl >= kMsMaxLevel) {
			if (leader) atomicExch(&ctl->err, BFS_EUNSUPPORTED);
			break;
		}
		if (lvl + 1 - base >= a.planes) {
			if (!levels) {  // planes kept for a later pass (betweenness): they must hold every level
				if (leader) atomicExch(&ctl->err, BFS_EUNSUPPORTED);
				break;
			}
			// planes full: write them out, keep the frontier's plane as plane 0
			if (!(ok = ms_spill(a, levels, ns, base, lvl, lev, epoch))) break;
			epoch += 2;
			base = lvl;
			if (leader) ctl->stats.spills++;
		}
		// the counters of the level after next are free again
		if (leader) {
			if (lvl < kMsTraceLevels) {
				ctl->stats.t_level[lvl] = global_timer_ns();
				ctl->stats.frontier[lvl] = nq + nb;
				ctl->stats.push[lvl] = qdeg * (unsigned long long) a.push_div < (unsigned long long) a.m;
			}
			MsCounters *c2 = &ctl->ctr[(lvl + 2) % 3];
			c2->nact = 0;
			c2->nbig = 0;
			c2->act_deg = 0;
			for (uint32_t k = 0; k < a.K; ++k) ctl->active[(lvl + 2) % 3][k] = 0;
		}
		if (threadIdx.x < 64) s_act[threadIdx.x] = 0;
		__syncthreads();
		// the sources with a frontier at this level (level 0: every source)
		const unsigned long long *act = lvl == 0 ? nullptr : ctl->active[lvl % 3];
		const uint64_t *cur = a.hist + (size_t) (lvl - base) * nK;
		uint64_t *nxt = a.hist + (size_t) (lvl + 1 - base) * nK;
		const uint64_t *actc = a.pmask + (size_t) (lvl - base) * a.n;
		uint64_t *actn = a.pmask + (size_t) (lvl + 1 - base) * a.n;
		unsigned long long *tph = lvl < kMsTraceLevels ? ctl->stats.t_phase[lvl] : nullptr;
		unsigned long long actdeg = 0;
		const bool masked = levels != nullptr && a.K > kMsRowWords;  // rows with an empty mask need no clearing
		const bool push = qdeg * (unsigned long long) a.push_div < (unsigned long long) a.m;
		if (push) {
			if (blockIdx.x == 0 && nb) ms_push_chunk_list(a, lvl, nb, wq);
			if (masked && nb <= kMsMarkBig && qdeg < a.n / kMsMarkDiv) ms_push_mark(a, lvl, nxt, nq, nb);
			else for (size_t i = t0; i < nK; i += stride) nxt[i] = 0;
			if (!(ok = grid_sync(ctl->bar, epoch, &ctl->err, a.wait_limit_ns, a.hold_barrier))) break;
			if (leader && tph) tph[0] = global_timer_ns();
			ms_push(a, lvl, cur, actc, nxt, nq, nb);
			if (!(ok = grid_sync(ctl->bar, epoch, &ctl->err, a.wait_limit_ns, a.hold_barrier))) break;
			if (leader && tph) tph[1] = global_timer_ns();
			ms_push_finish(a, lvl, nxt, actn, actdeg, s_act);
		} else {
			const MsPull p{cur, actc, nxt, actn, act, &ctl->ctr[(lvl + 1) % 3], a.queue[(lvl + 1) & 1],
					masked};
			ms_pull<KK>(a, p, &ctl->work[lvl], actdeg, gathered, wq, s_act);
		}
		// the next frontier's out-degree: per-CTA sum, one atomic per CTA
		const unsigned long long d = warp_sum(actdeg);
		if (lane_id() == 0) red[warp_id()] = d;
		__syncthreads();
		if (threadIdx.x == 0) {
			unsigned long long tsum = 0;
			for (int w = 0; w < kMsWarps; ++w) tsum += red[w];
			if (tsum) atomicAdd(&ctl->ctr[(lvl + 1) % 3].act_deg, tsum);
			if (blockIdx.x == 0) {
				ctl->stats.levels = lvl + 1;
				if (push) ctl->stats.push_levels++;
			}
		}
		// the next level's active sources: this CTA's share
		if (threadIdx.x < a.K && s_act[threadIdx.x])
			atomicOr(&ctl->active[(lvl + 1) % 3][threadIdx.x], s_act[threadIdx.x]);
		__syncthreads();
		ok = grid_sync(ctl->bar, epoch, &ctl->err, a.wait_limit_ns, a.hold_barrier);
	}
	if (leader) {
		ctl->stats.t_levels1 = global_timer_ns();
		if (lvl < kMsTraceLevels) ctl->stats.t_level[lvl] = ctl->stats.t_levels1;
		ctl->stats.base = base;
		ctl->stats.complete = complete ? 1u : 0u;
	}
	if (complete) {
		// TEPS numerator: sum over (source, reached vertex) of out-degree
		unsigned long long tr = 0;
		for (uint32_t v = t0; v < a.n; v += stride) {
			uint32_t c = 0;
			for (uint32_t k = 0; k < a.K; ++k) c += __popcll(ld_cg64(a.vis + (size_t) v * a.K + k));
			tr += (unsigned long long) c * deg_of(a, v);
		}
		tr = warp_sum(tr);
		__syncthreads();
		if (lane_id() == 0) red[warp_id()] = tr;
		__syncthreads();
		if (threadIdx.x == 0) {
			unsigned long long tsum = 0;
			for (int w = 0; w < kMsWarps; ++w) tsum += red[w];
			if (tsum) atomicAdd(&ctl->stats.traversed, tsum);
		}
	}
	const unsigned long long gw = warp_sum(gathered);
	if (lane_id() == 0 && gw) atomicAdd(&ctl->stats.edges, gw);
	if (leader) ctl->stats.depth = lvl;
}

// The final output pass, its own launch after k_ms_bfs.  Plane depth - base is
// the empty frontier; after an early output pass, plane 0 was written too.  A
// tile is kW words wide, a thread per (vertex, word): with one or two words per
// vertex, tiles of four would leave most threads idle.  512 threads: level rows
// go out in pieces of 128 bytes or more, 5.5 ms for 2^22 vertices and 4,096
// sources (17 GB of levels, 4 TB/s with the planes read; 11.7 ms before the words
// came ahead and by permute), where pieces of 64 bytes (256 threads, option
// batch_output_tile) take 7.3 and of 256 bytes (1,024) 5.9.
template <int kThreads, uint32_t kW, bool kShift>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 4 : 2) k_ms_emit(MsArgs a, uint32_t ns, uint8_t *levels) {
	constexpr uint32_t kV = kThreads / kW;
	extern __shared__ __align__(16) uint8_t lev[];
	const MsStats &st = a.ctl->stats;
	if (!st.complete) return;
	const uint32_t base = st.base, depth = st.depth;
	const uint32_t first = base == 0 ? 0 : 1;
	if (depth < base + first + 1) return;
	ms_emit<true, kV, kW, kShift>(a, levels, ns, base, first, depth - 1 - base, base != 0, lev);
}

// The output pass's launch for a tile of kThreads / kW vertices x kW words.
template <int kThreads, uint32_t kW, bool kShift>
int emit_launch(const MsArgs &a, uint32_t ns, uint8_t *levels, int num_sms, cudaStream_t st) {
	constexpr int kBytes = (int) emit_bytes(kThreads / kW, kW, true);
	auto fn = k_ms_emit<kThreads, kW, kShift>;
	if (kBytes > 48 * 1024 && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) != cudaSuccess)
		return BFS_ECUDA;
	int per_sm = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, kBytes) != cudaSuccess || per_sm < 1)
		return BFS_ECUDA;
	fn<<<num_sms * per_sm, kThreads, kBytes, st>>>(a, ns, levels);
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

// chunk_slot[c]: the index of chunk c's destination in in_big (ascending).
__global__ void k_ms_chunk_slots(const uint32_t *chunk_v, uint32_t nchunks, const uint32_t *in_big, uint32_t nbig,
		uint32_t *chunk_slot) {
	for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nchunks; c += gridDim.x * blockDim.x) {
		const uint32_t v = chunk_v[c];
		uint32_t lo = 0, hi = nbig - 1;
		while (lo < hi) {
			const uint32_t mid = (lo + hi) / 2;
			if (in_big[mid] < v) lo = mid + 1;
			else hi = mid;
		}
		chunk_slot[c] = lo;
	}
}

int ms_chunk_slots(const uint32_t *chunk_v, uint32_t nchunks, const uint32_t *in_big, uint32_t nbig, uint32_t *chunk_slot) {
	if (!nchunks || !nbig) return BFS_OK;
	k_ms_chunk_slots<<<std::min<uint32_t>((nchunks + 255) / 256, 1024), 256>>>(chunk_v, nchunks, in_big, nbig, chunk_slot);
	return cudaGetLastError() == cudaSuccess && cudaStreamSynchronize(0) == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

int ms_launch(const MsArgs &a, const uint32_t *d_sources, uint32_t ns, uint8_t *levels, int num_sms, cudaStream_t st,
		int *grid, cudaEvent_t between, cudaEvent_t between2) {
	static_assert(kMsRowWords == 4, "a kernel for each");
	const auto fn = a.K == 1 ? k_ms_bfs<1> : a.K == 2 ? k_ms_bfs<2> : a.K == 3 ? k_ms_bfs<3> : a.K == 4 ? k_ms_bfs<4>
			: a.K <= 8 ? k_ms_bfs<8> : a.K <= 16 ? k_ms_bfs<16> : a.K <= kGroupMaxWords ? k_ms_bfs<kGroupMaxWords> : k_ms_bfs<kMsMaxWords>;
	int per_sm = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kMsThreads, 0) != cudaSuccess || per_sm < 1)
		return BFS_ECUDA;
	const uint64_t state = a.K <= kMsRowWords ? (uint64_t) a.n * a.K : ~0ull;
	per_sm = std::min(per_sm, a.ctas_per_sm ? (int) a.ctas_per_sm : state <= kMsSmallState ? 1 : 2);
	const int ctas = !a.ctas_per_sm && state <= kMsTinyState ? std::max(num_sms / 2, 1) : num_sms * per_sm;
	if (grid) *grid = ctas;
	if (cudaMemsetAsync(a.ctl, 0, sizeof(MsControl), st) != cudaSuccess) return BFS_ECUDA;
	MsArgs aa = a;
	// the pull's items: see ms_pull
	const uint32_t nwarps = (uint32_t) ctas * kMsWarps;
	aa.run = 1;
	aa.blk_shift = 5;
	if (a.K <= kMsRowWords) {
		aa.run = std::min(std::max(a.nchunks / (nwarps * 2), 1u), kMsRun);
	} else {
		while (aa.blk_shift > 2 && a.n >> aa.blk_shift < kMsBlocks * nwarps) --aa.blk_shift;
		while (aa.blk_shift > 0 && a.n >> aa.blk_shift < nwarps / 2) --aa.blk_shift;
	}
	aa.nruns = (a.nchunks + aa.run - 1) / aa.run;
	const uint32_t nblk = (uint32_t) (((uint64_t) a.n + (1u << aa.blk_shift) - 1) >> aa.blk_shift);
	uint32_t blocks = 1;
	while (a.K <= kMsRowWords && blocks < kMsMaxClaim && nblk / (2 * blocks) >= nwarps * kMsClaims) blocks *= 2;
	aa.claim = blocks << aa.blk_shift;
	aa.nclaims = (nblk + blocks - 1) / blocks;
	const uint32_t *src = d_sources;
	uint32_t nsrc = ns;
	uint8_t *out = levels;
	void *args[] = {&aa, (void *) &src, &nsrc, &out};
	if (cudaLaunchCooperativeKernel((const void *) fn, dim3(ctas), dim3(kMsThreads), args, 0, st) !=
			cudaSuccess)
		return BFS_ECUDA;
	if (between && cudaEventRecord(between, st) != cudaSuccess) return BFS_ECUDA;
	if (between2 && cudaEventRecord(between2, st) != cudaSuccess) return BFS_ECUDA;
	if (levels) {
		const uint32_t words = a.out_tile || a.K > 2 ? kEmitW : a.K;  // an explicit tile width is one of four-word tiles
		const bool shift = a.n % 16 != 0 || (uintptr_t) levels % 16 != 0;
		const auto launch = words == 1 ? (shift ? emit_launch<512, 1, true> : emit_launch<512, 1, false>)
				: words == 2 ? (shift ? emit_launch<512, 2, true> : emit_launch<512, 2, false>)
				: a.out_tile == 64 ? (shift ? emit_launch<256, kEmitW, true> : emit_launch<256, kEmitW, false>)
				: (shift ? emit_launch<512, kEmitW, true> : emit_launch<512, kEmitW, false>);
		const int rc = launch(a, ns, levels, num_sms, st);
		if (rc) return rc;
	}
	return cudaGetLastError() == cudaSuccess ? BFS_OK : BFS_ECUDA;
}

} // namespace bfsg
