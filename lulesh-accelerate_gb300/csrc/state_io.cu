// state_io.cu -- the Domain record of a small mesh between the host and the
// device arrays, and the scalars that the host sets.
//
// A copy command costs 2-3 us of its own on the copy engine, and 8 from or to
// pageable memory: eleven of them are most of a state transfer below 10^4
// nodes (s=8: 28 us from pinned memory, 89 us to pageable memory).  A small
// state instead passes through a buffer of mapped pinned memory, which one
// kernel reads or writes directly: 17 us up, 12 us down, and a memory copy on
// the host, ~35 us per MB.  A larger state in pinned arrays goes the same way
// without the buffer: the kernel reads or writes the host's own arrays, 22 us
// against the copy engine's 42 at s=30, 57 against 75 at s=47, 2.99 ms against
// 3.01 at s=192 (205 GB/s, the link's rate).
// The scalars go by value with the launch, where reading them back, changing
// them and writing them took two copies and two waits (17 us, 9 now).
#include "lulesh_internal.h"
#include "kernels.h"

#include <cuda_runtime.h>

namespace lulesh {

namespace {

__device__ void set_scalars(DevScalars *sc, const ScalarSet &v)
{
    if (v.clock) {
        sc->time = v.time;
        sc->deltatime = v.deltatime;
    }
    if (v.constraints) {
        sc->dtcourant = v.dtcourant;
        sc->dthydro = v.dthydro;
        sc->cycle = v.cycle;
        sc->courant_key = ~0ULL;
        sc->hydro_key = ~0ULL;
    }
    // an error stops a kinematics launch part way: what it kept is of two states
    if (v.moved || sc->err_any) sc->geo_valid = 0;
    sc->err_any = 0;
    for (int i = 0; i < ERR_NUM; ++i) sc->err[i] = 0;
}

// Value t of the state: six node fields of nn values, then five element
// fields of ne, in the order of StateView::field.
struct Place {
    int field, i;
};
__device__ __forceinline__ Place place_of(const StateView &v, int t)
{
    const int nodes = 6 * v.nn;
    const int f = t < nodes ? t / v.nn : 6 + (t - nodes) / v.ne;
    return {f, t < nodes ? t - f * v.nn : (t - nodes) - (f - 6) * v.ne};
}

__global__ void __launch_bounds__(256) k_state_in(const __grid_constant__ StateView v, const double *stage, int total,
                                                  DevScalars *sc, const __grid_constant__ ScalarSet set)
{
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t == 0) set_scalars(sc, set);
    if (t >= total) return;
    const Place at = place_of(v, t);
    if ((v.present >> at.field) & 1) v.field[at.field][at.i] = stage[t];
}

__global__ void __launch_bounds__(256) k_state_out(const __grid_constant__ StateView v, double *stage, int total,
                                                   const DevScalars *sc, DevScalars *host_sc)
{
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t == 0) *host_sc = *sc;
    if (t >= total) return;
    const Place at = place_of(v, t);
    if ((v.present >> at.field) & 1) stage[t] = v.field[at.field][at.i];
}

// One field per blockIdx.y, kPerThread values per thread, all loaded before any
// is stored: the link's latency is ~2 us.
constexpr int kPerThread = 4;
template <bool kIn>
__device__ __forceinline__ void copy_field(const StateView &v, const HostState &host)
{
    const int f = blockIdx.y, n = f < 6 ? v.nn : v.ne;
    if (!((v.present >> f) & 1)) return;
    double *to = kIn ? v.field[f] : host.field[f];
    const double *from = kIn ? host.field[f] : v.field[f];
    const long first = (long)blockIdx.x * (256 * kPerThread) + threadIdx.x;
    double x[kPerThread];
#pragma unroll
    for (int i = 0; i < kPerThread; ++i)
        if (first + 256 * i < n) x[i] = from[first + 256 * i];
#pragma unroll
    for (int i = 0; i < kPerThread; ++i)
        if (first + 256 * i < n) to[first + 256 * i] = x[i];
}

__global__ void __launch_bounds__(256) k_state_from_host(const __grid_constant__ StateView v, const __grid_constant__ HostState host,
                                                         DevScalars *sc, const __grid_constant__ ScalarSet set)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) set_scalars(sc, set);
    copy_field<true>(v, host);
}

__global__ void __launch_bounds__(256) k_state_to_host(const __grid_constant__ StateView v, const __grid_constant__ HostState host,
                                                       const DevScalars *sc, DevScalars *host_sc)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *host_sc = *sc;
    copy_field<false>(v, host);
}

// Wide enough for the longest field: a mesh given by its lists may have more
// elements than nodes.
dim3 field_grid(const StateView &v)
{
    const long n = v.nn > v.ne ? v.nn : v.ne;
    return dim3((unsigned)((n + 256L * kPerThread - 1) / (256L * kPerThread)), 11);
}

}  // namespace

void launch_state_from_host(const StateView &v, const HostState &host, DevScalars *sc, const ScalarSet &set, cudaStream_t st)
{
    k_state_from_host<<<field_grid(v), 256, 0, st>>>(v, host, sc, set);
}

void launch_state_to_host(const StateView &v, const HostState &host, const DevScalars *sc, DevScalars *host_sc, cudaStream_t st)
{
    k_state_to_host<<<field_grid(v), 256, 0, st>>>(v, host, sc, host_sc);
}

void launch_set_scalars(DevScalars *sc, const ScalarSet &set, cudaStream_t st)
{
    k_state_in<<<1, 256, 0, st>>>(StateView{}, nullptr, 0, sc, set);
}

void launch_state_in(const StateView &v, const double *stage, DevScalars *sc, const ScalarSet &set, cudaStream_t st)
{
    const int total = 6 * v.nn + 5 * v.ne;
    k_state_in<<<(total + 255) / 256, 256, 0, st>>>(v, stage, total, sc, set);
}

void launch_state_out(const StateView &v, double *stage, const DevScalars *sc, DevScalars *host_sc, cudaStream_t st)
{
    const int total = 6 * v.nn + 5 * v.ne;
    k_state_out<<<(total + 255) / 256, 256, 0, st>>>(v, stage, total, sc, host_sc);
}

}  // namespace lulesh
