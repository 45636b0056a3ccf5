// build_device.h -- kernels that build a graph's device layout from an edge
// list (build_device.cu).  Internal.
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace bfsg {

struct DeviceBuildShape {
	uint32_t w, s, stripes;
	uint32_t vbits, cbits;
};

// out_deg[u]++ / in_deg[v]++ per edge (both zeroed by the caller); an id
// >= n sets *err to BFS_EFORMAT.
int dbuild_degrees(const uint32_t *src, const uint32_t *dst, uint64_t m, uint32_t n, uint32_t *out_deg,
		uint32_t *in_deg, int *err, int num_sms, cudaStream_t st);
// out[0..n] = exclusive prefix sums of in[0..n) (out[n] = total); tmp holds
// dbuild_scan_tmp_words(n) words.
uint32_t dbuild_scan_tmp_words(uint32_t n);
int dbuild_exclusive_scan(const uint32_t *in, uint32_t n, uint32_t *tmp, uint32_t *out, cudaStream_t st);
// out[cursor[key[i]]++] = val[i]
int dbuild_scatter(const uint32_t *key, const uint32_t *val, uint64_t m, uint32_t *cursor, uint32_t *out, int num_sms,
		cudaStream_t st);
// From the degrees: the has-in-edge bitmap, per vertex the batched pull's
// chunks of `chunk` in-edges (0 up to `big` of them) and whether there are
// any, and the largest out-degree (*max_degree zeroed by the caller).
int dbuild_vertex_facts(const uint32_t *out_deg, const uint32_t *in_deg, uint32_t n, uint32_t big, uint32_t chunk,
		uint32_t *hasin, uint32_t *chunks, uint32_t *is_big, uint32_t *max_degree, int num_sms, cudaStream_t st);
// Per vertex of the lists `off`, its chunks in batched betweenness (bb_chunk_len; 0 up to `chunk` edges).
int dbuild_chunk_counts(const uint32_t *off, uint32_t n, uint32_t chunk, uint32_t *chunks, int num_sms, cudaStream_t st);
// The batched pull's lists from the exclusive scans of is_big and chunks; with
// big_off null the chunks of batched betweenness alone (of any lists, in_off).
int dbuild_big_lists(uint32_t n, const uint32_t *big_off, const uint32_t *chunk_off, const uint32_t *in_off,
		uint32_t nchunks, uint32_t chunk, uint32_t *in_big, uint32_t *chunk_v, uint32_t *chunk_beg, int num_sms,
		cudaStream_t st);
// The blocks of kPullBlock words of the has-in-edge bitmap that have a bit, in
// order, and their number (one CTA).
int dbuild_pull_blocks(const uint32_t *hasin, uint32_t nwords, uint32_t *blocks, uint32_t *count, cudaStream_t st);
// in-edges per tile column
int dbuild_col_edges(const uint32_t *in_off, uint32_t n, uint32_t w, uint32_t side, uint32_t *col_edges, cudaStream_t st);

// A run of one column group's in-edges, the work of one CTA.
struct SegItem {
	uint32_t group, beg, end;
};
// Whether a CTA can count this many stripes in shared memory; graphs with more
// take the per-edge dbuild_seg_hist and dbuild_seg_fill.
bool dbuild_seg_items_fit(uint32_t stripes);
std::vector<SegItem> dbuild_seg_items(const std::vector<uint32_t> &group_col, const std::vector<uint64_t> &col_edges);
// dbuild_seg_hist and dbuild_seg_fill from the in-edge lists
int dbuild_seg_count(const uint32_t *in_src, const SegItem *items, uint32_t num_items, uint32_t sw, uint32_t stripes,
		uint32_t *seg_count, cudaStream_t st);
int dbuild_seg_pack(const uint32_t *in_off, const uint32_t *in_src, const SegItem *items, uint32_t num_items,
		const DeviceBuildShape &sh, const uint32_t *group_col, uint32_t n, uint32_t *cursor, uint32_t *words, cudaStream_t st);
// edges per packed segment (group(v) * stripes + stripe(u)), zeroed by the caller
int dbuild_seg_hist(const uint32_t *src, const uint32_t *dst, uint64_t m, const DeviceBuildShape &sh,
		const uint32_t *group_of, uint32_t *seg_count, int num_sms, cudaStream_t st);
// packed words into their segments (cursor = a copy of the segment offsets)
int dbuild_seg_fill(const uint32_t *src, const uint32_t *dst, uint64_t m, const DeviceBuildShape &sh,
		const uint32_t *group_of, const uint32_t *group_col, uint32_t *cursor, uint32_t *words, int num_sms,
		cudaStream_t st);
// padding words after each segment's edges
int dbuild_seg_pad(const uint32_t *seg_off, const uint32_t *seg_count, uint64_t nseg, uint32_t stripes,
		const uint32_t *pad_word, uint32_t *words, int num_sms, cudaStream_t st);

} // namespace bfsg
