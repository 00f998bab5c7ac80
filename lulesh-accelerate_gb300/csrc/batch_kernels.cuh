// batch_kernels.cuh -- persistent kernels over the active tiles of one size
// class of a batched ensemble.  Each block walks the class's active-tile list
// with a grid stride; a tile is kTile consecutive elements (nodes) of one
// instance, processed blockDim at a time (kTile / blockDim elements per
// thread).  The per-element work is the single-instance body, given the
// instance's scalar block.
#pragma once

#include "common.cuh"

namespace lulesh {

// The block's shares of the active tiles, one element (node) per thread: a
// tile is kTile / blockDim shares, dealt to the blocks with a grid stride.
// The first share's list entry is loaded together with the list's length (a
// launch has no more blocks than the class has shares, so the entry exists,
// whatever it holds).  visit(tile, i): i the thread's place, past the tile's
// end or not.
template <class Visit>
__device__ __forceinline__ void for_active_tiles(const int *count, const ActiveTile *list, Visit &&visit)
{
    const int shares = kTile / blockDim.x;   // blockDim: 32, 64, 128, 256, or a multiple of 32 with a remainder
    const int per = shares * blockDim.x == kTile ? shares : shares + 1;
    ActiveTile a = list[blockIdx.x / per];
    const int n = *count * per;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        if (i != (int)blockIdx.x) a = list[i / per];
        const int o = (i % per) * blockDim.x + threadIdx.x;
        visit(a, o < kTile ? a.begin + o : a.end);
    }
}

template <void (*Body)(const Dom &, int, DevScalars *)>
__device__ __forceinline__ void kb_elem_tiles(const Dom &d, const BatchView &b, int cls)
{
    for_active_tiles(b.counts + cls, b.active_etiles + b.eclass_off[cls], [&](const ActiveTile &a, int k) {
        DevScalars *sc = d.sc + a.inst;
        if (k < a.end && !sc->err_any) Body(d, k, sc);
    });
}

// The material kernel also reduces the instance's constraint keys: one
// block minimum per share (every thread reaches the barrier; the trip counts
// are uniform over the block).
template <void (*Body)(const Dom &, int, DevScalars *, unsigned long long &, unsigned long long &)>
__device__ __forceinline__ void kb_material_tiles(const Dom &d, const BatchView &b, int cls)
{
    for_active_tiles(b.counts + cls, b.active_etiles + b.eclass_off[cls], [&](const ActiveTile &a, int k) {
        DevScalars *sc = d.sc + a.inst;
        unsigned long long kc = ~0ULL, kh = ~0ULL;
        if (k < a.end && !sc->err_any) Body(d, k, sc, kc, kh);
        block_min_publish(kc, kh, sc);
        __syncthreads();   // the shared staging of block_min_publish is reused next share
    });
}

// kRegs: the registers of a thread, so that a kernel keeps the resident warps
// of the single-instance one whatever the loop around the body costs (the
// double-float force body at 178 instead of 168 has two 128-thread blocks per
// SM instead of three: 114 us against 90 at 77^3 elements).
template <void (*Body)(const Dom &, int, DevScalars *), int kRegs>
__global__ void __maxnreg__(kRegs) kb_elem(const __grid_constant__ Dom d, const __grid_constant__ BatchView b, int cls)
{
    kb_elem_tiles<Body>(d, b, cls);
}

template <void (*Body)(const Dom &, int, DevScalars *, unsigned long long &, unsigned long long &)>
__global__ void kb_material(const __grid_constant__ Dom d, const __grid_constant__ BatchView b, int cls)
{
    kb_material_tiles<Body>(d, b, cls);
}

// Register-capped variants for the kinematics and material bodies, which
// wait on their gathers: blocks of up to kBatchMaxBlock threads (the
// autotuner's largest), kMinBlocks of them resident per SM, so 4 -> 64
// registers, 3 -> 85 and 2 -> 128.  The material bodies of both arithmetics
// run at 64 (as the single-instance material kernels do).  On the
// 528-instance split ensemble (kinematics at 128 registers instead of 134,
// material at 64 instead of 77) this took 36.7 s to 30.2 s; capping the
// force body as well (64 or 85 registers, with spills) lost 5 %.
constexpr int kBatchMaxBlock = 256;

template <void (*Body)(const Dom &, int, DevScalars *), int kMinBlocks>
__global__ void __launch_bounds__(kBatchMaxBlock, kMinBlocks)
    kb_elem_capped(const __grid_constant__ Dom d, const __grid_constant__ BatchView b, int cls)
{
    kb_elem_tiles<Body>(d, b, cls);
}

template <void (*Body)(const Dom &, int, DevScalars *, unsigned long long &, unsigned long long &),
          int kMinBlocks>
__global__ void __launch_bounds__(kBatchMaxBlock, kMinBlocks)
    kb_material_capped(const __grid_constant__ Dom d, const __grid_constant__ BatchView b, int cls)
{
    kb_material_tiles<Body>(d, b, cls);
}

template <void (*Body)(const Dom &, int, const DevScalars *), int kRegs>
__global__ void __maxnreg__(kRegs) kb_node(const __grid_constant__ Dom d, const __grid_constant__ BatchView b, int cls)
{
    for_active_tiles(b.counts + kMaxClasses + cls, b.active_ntiles + b.nclass_off[cls], [&](const ActiveTile &a, int n) {
        const DevScalars *sc = d.sc + a.inst;
        if (n >= a.end || sc->err_any) return;
        // the instance's positions move: its geometry cache goes stale (one
        // store: every block's would keep taking the line away from the
        // others' loads of the scalars, 115 us instead of 35 at 78^3 nodes)
        if (d.geo && n == sc->node_begin) d.sc[a.inst].geo_valid = 0;
        Body(d, n, sc);
    });
}

}  // namespace lulesh
