// kernels_api.h -- host-side entry points of bfs_kernels.cu (internal).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/bfs_gb300.h"
#include "bfs_device.cuh"

namespace bfsg {

constexpr uint32_t kSentinelWord = 0xFFFFFFFFu;
constexpr uint32_t kUnvisitedWord = 0xFFFFFFFFu;
constexpr uint32_t kMaxSliceBatch = 16;   // frontier slices staged together by the bottom-up step
constexpr uint32_t kSliceBudgetWords = 8192;
// Bulk-copy pipeline of the bottom-up step: stages per CTA, packed words per
// stage and the shared-memory budget of the frontier slices of one stage.
constexpr uint32_t kTmaStages = 3;
constexpr uint32_t kTmaEdgeWords = 4096;
constexpr uint32_t kTmaSliceWords = 4096;

enum StepKind { kStepSeed = 0, kStepClear, kStepToDense, kStepToSparse, kStepExpand, kStepDense };

// Top-down steps that one CTA takes in a row while the rest of the grid waits at
// one barrier: at most kSoloLevels, and no more than fit a quarter of the wait
// limit at kSoloStepNs, the longest seen (layers of 40 vertices, 1,600 edges a step:
// 128 steps are 0.99 ms, and a limit of 0.5 ms ran out in a sound traversal).
constexpr uint32_t kSoloLevels = 128, kSoloStepNs = 16000;
inline uint32_t solo_levels(uint64_t wait_limit_ns) {
	const uint64_t fit = wait_limit_ns / (4 * kSoloStepNs);
	return fit < kSoloLevels ? (uint32_t) fit : kSoloLevels;
}
// The cooperative grid at full occupancy and the dynamic shared memory of a
// traversal whose bottom-up steps are `bottom_up` (BFS_BU_*).
int persistent_grid(const DevGraph &g, uint32_t batch, uint32_t bottom_up, int device, int num_sms, int *grid, size_t *smem);
// Clears the run state for the stepwise mode (the persistent kernel clears
// and seeds by itself).
int launch_init(const DevGraph &g, const RunCtx &r, cudaStream_t st, int num_sms);
int launch_persistent(const DevGraph &g, const RunCtx &r, const StepParams &p, uint32_t batch, int grid,
		size_t smem, cudaStream_t st);
// The one-cluster traversal (bfs_cluster.cu): CTAs of its cluster for a graph,
// 0 where the graph is too large for it (or the device takes no such cluster).
// Up to kClusterDenseVertices; above, up to kClusterMaxVertices, only with at most
// kClusterSparseDegree edges a vertex (many levels of few edges): the pulls of
// denser ones want more than 16 SMs.  Both limits were found on dense graphs; a
// street grid was measured at one size, and its own limit is higher (90,000 vertices, 2^21 edges: rmat 102 us in
// the cluster, 98 on the grid; 2^20 edges: rmat 107 and 91, uniform 120 and 108; a
// street grid of 90,000: 728 and 923; 2^16 vertices, 2^20 edges: rmat 81 and 82,
// 2^15 vertices 59 and 77).
constexpr uint32_t kClusterDenseVertices = 1u << 16, kClusterSparseDegree = 4;
constexpr uint32_t kClusterMaxVertices = 3u << 15;
constexpr uint32_t kClusterMaxEdges = 1u << 24;
constexpr uint32_t kClusterVerticesPerCta = 1024;
int cluster_ctas(const DevGraph &g);
int launch_cluster(const DevGraph &g, const RunCtx &r, const StepParams &p, int ctas, cudaStream_t st);
int launch_step(int kind, const DevGraph &g, const RunCtx &r, const StepParams &p, uint32_t step,
		uint32_t batch, int grid, size_t smem, cudaStream_t st);
int kernel_threads();

} // namespace bfsg
