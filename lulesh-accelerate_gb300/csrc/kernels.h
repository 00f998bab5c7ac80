// kernels.h -- launchers of the step kernels (host side of the .cu files).
#pragma once

#include "lulesh_internal.h"

#include <cuda_runtime.h>

namespace lulesh {

// Threads per block of the element and node kernels.  The element kernels
// are bound by instruction issue at 64-168 registers; 128 threads give two
// to eight resident blocks per SM at their register counts (the kinematics
// kernels run two such blocks' worth as one, see kin_block).  The node
// updates, gathers bound by memory, ran 1-2 % faster in 128-thread blocks
// than in 256 (512: 2-3 % slower).
constexpr int kBlockElem = 128;
constexpr int kBlockNode = 128;

inline int elem_block(const Dom &d) { return d.eblock ? d.eblock : kBlockElem; }
inline int node_block(const Dom &d) { return d.nblock ? d.nblock : kBlockNode; }

// The kinematics kernels (128 registers, two 256-thread blocks per SM
// rather than four of 128: the same sixteen warps, but each SM sub-partition
// runs two warps of one block, which start together and walk the long
// straight-line body close to each other, so fewer warps wait on
// instruction fetch): 4-6 % faster at s=192 in both arithmetics.
constexpr int kKinBlockFactor = 2;
inline int kin_block(const Dom &d) { return kKinBlockFactor * elem_block(d); }
// The material kernels (64 registers, 1024 threads per SM in any split) take
// larger blocks on larger meshes for the same reason: their waits for
// instructions were a fifth of a warp's time.  s=192: plain 528 us in blocks
// of 128 threads, 514 of 256, 495 of 512 (and 4 % more than that in one of
// 1024), split 492, 473, 465; s=96 77, 74, 74 and 72, 69, 69; s=47, with too
// few blocks to spread, 15, 15, 17.
constexpr int kMatBlockFactor = 4;
inline int mat_block(const Dom &d)
{
    return elem_block(d) * (d.ne >= 1000000 ? kMatBlockFactor : d.ne >= 100000 ? 2 : 1);
}
// Block sizes for a mesh of ne elements and nn nodes on a GPU with sms SMs:
// the defaults, halved (down to one warp) while a kernel would have fewer
// than four blocks per SM -- one FP64-bound element per thread makes the SM
// with one block more than its neighbours the one that sets the time.
inline void choose_blocks(Dom &d, int sms)
{
    int eb = kBlockElem, nb = kBlockNode;
    while (eb > 32 && (d.ne + eb - 1) / eb < 4L * sms) eb /= 2;
    while (nb > 32 && (d.nn + nb - 1) / nb < 4L * sms) nb /= 2;
    d.eblock = eb;
    d.nblock = nb;
}

struct CycleEnd;   // common.cuh
void launch_end_cycle(const Dom &d, cudaStream_t st, const CycleEnd &end);

// The initial state and mesh data of one cube, or of a batch's cubes with
// their tiles' numbers (mesh_gpu.cu), into arrays that hold zeros.
void launch_build_cube(const Dom &d, const CubeDesc &cube, cudaStream_t st);
void launch_build_cubes(const Dom &d, const CubeDesc *cubes, const int *etile_cube, const int *ntile_cube, cudaStream_t st);

// The scalars that a call sets, beside clearing the error words.
struct ScalarSet {
    double time, deltatime, dtcourant, dthydro;
    int cycle;
    bool clock;         // time and deltatime
    bool constraints;   // dtcourant, dthydro and the cycle count; the minima start afresh
    bool moved;         // new positions or velocities: the geometry cache is stale
};
// The fields of the Domain record in the order of lulesh_upload_domain, and
// which of them a call transfers (bit f).
struct StateView {
    double *field[11];
    int nn, ne;
    unsigned present;
};
// The device addresses of the host's arrays, where all of them are pinned.
struct HostState {
    double *field[11];
};
void launch_set_scalars(DevScalars *sc, const ScalarSet &set, cudaStream_t st);
// A state between its fields and the host's own pinned arrays
void launch_state_from_host(const StateView &v, const HostState &host, DevScalars *sc, const ScalarSet &set, cudaStream_t st);
void launch_state_to_host(const StateView &v, const HostState &host, const DevScalars *sc, DevScalars *host_sc, cudaStream_t st);
// A whole state between its fields and a mapped host buffer that holds them
// one after the other (state_io.cu)
void launch_state_in(const StateView &v, const double *stage, DevScalars *sc, const ScalarSet &set, cudaStream_t st);
void launch_state_out(const StateView &v, double *stage, const DevScalars *sc, DevScalars *host_sc, cudaStream_t st);

// Plain FP64 path (step_fp64.cu).
void launch_time_increment(const Dom &d, cudaStream_t st);
void launch_lagrange_nodal(const Dom &d, cudaStream_t st);
// end null: without the time constraints
void launch_lagrange_elements(const Dom &d, cudaStream_t st, const CycleEnd *end);
void launch_time_constraints(const Dom &d, cudaStream_t st);
void launch_run_prologue(const Dom &d, cudaStream_t st, const int *max_cycles,
                         cudaGraphConditionalHandle h, int *active);
void launch_run_body(const Dom &d, cudaStream_t st, cudaGraphConditionalHandle h, int *active);
int kernels_per_cycle();
constexpr int kRunCycleLimit = LULESH_RUN_CYCLE_BUDGET;
// time increment, force, node, kinematics, material, constraint publication
constexpr int kTimedKernels = 6;
void launch_cycle_timed(const Dom &d, cudaStream_t st, cudaEvent_t ev[kTimedKernels + 1]);
// The accessors' conversions of a pair field (step_df.cu): a pair is its
// exact sum, a double its FP32 rounding and the remainder's.
void launch_pairs_to_doubles(const double *pairs, double *out, long n, cudaStream_t st);
void launch_doubles_to_pairs(const double *in, double *pairs, long n, cudaStream_t st);
// lulesh_probe_pairs (step_df.cu)
void launch_pair_probe(double *sums, unsigned long long *worst, int n, cudaStream_t st);
void launch_fp64_probe(double *out, int blocks, int threads, int iters, cudaStream_t st);
void launch_rate_probe(int which, float *out, int blocks, int threads, int iters, cudaStream_t st);
// largest relative differences (as order keys of non-negative doubles) of the
// library's inverse cube root and square root from CUDA's, over n arguments
void launch_math_probe(unsigned long long *keys, int n, cudaStream_t st);

// The plain path's double-float element kernels (step_df.cu); the launchers
// above call them when Dom::df is set.
void launch_elem_force_df(const Dom &d, cudaStream_t st);
void launch_node_update_df(const Dom &d, cudaStream_t st);
void launch_elem_kinematics_df(const Dom &d, cudaStream_t st);
void launch_elem_material_df(const Dom &d, cudaStream_t st, const CycleEnd *end);
void launch_batch_kernel_df(const Dom &d, const BatchView &b, cudaStream_t st, int kernel, int cls, LaunchCfg cfg);
int batch_max_blocks_df(int kernel, int block, bool early);

// Split-precision path (step_split.cu).
void launch_split_sync(const Dom &d, cudaStream_t st);
void launch_lagrange_nodal_split(const Dom &d, cudaStream_t st);
void launch_lagrange_elements_split(const Dom &d, cudaStream_t st, const CycleEnd *end);
void launch_run_body_split(const Dom &d, cudaStream_t st, cudaGraphConditionalHandle h, int *active);
void launch_cycle_timed_split(const Dom &d, cudaStream_t st, cudaEvent_t ev[kTimedKernels + 1]);

// Batched ensembles (batch.cu drives these; kernel ids 0..3 = force, node
// update, kinematics, material).
void launch_batch_kernel_fp64(const Dom &d, const BatchView &b, cudaStream_t st, int kernel, int cls,
                              LaunchCfg cfg);
void launch_batch_kernel_split(const Dom &d, const BatchView &b, cudaStream_t st, int kernel, int cls,
                               LaunchCfg cfg);
int batch_max_blocks_fp64(int kernel, int block, int arith, bool early);
int batch_max_blocks_split(int kernel, int block, bool early);
void launch_batch_force_split_staged(const Dom &d, const BatchView &b, const StagedClass &sc, int rows,
                                     LaunchCfg cfg, cudaStream_t st);
int batch_max_blocks_split_staged(int rows);

}  // namespace lulesh
