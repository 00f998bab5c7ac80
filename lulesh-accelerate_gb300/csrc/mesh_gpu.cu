// mesh_gpu.cu -- the Sedov problem on s^3 cubes, set up on the device.
//
// What HostMesh::build (mesh.cpp) makes on the host -- coordinates,
// connectivity, boundary bits, reference volumes and masses, the initial
// energy -- written straight into the device arrays, to the same bits: the
// floating-point work is one rounded operation at a time in the host's
// order.  Two kernels, an element and then a node per thread, for one cube or
// for all cubes of a batch.  They write ~150 bytes an element and end within
// a fraction of a millisecond; on the host the lists' construction, their
// renumbering and the copies of sixteen arrays per cube took 60-70 ns an
// element (476k elements in eight cubes: 30 ms of a 118 ms ensemble run of
// 300 cycles).  The node-to-corner and face-neighbour lists are not made at
// all: on a cube every kernel forms them from the indices.
#include "lulesh_internal.h"
#include "kernels.h"
#include "elem_volume.h"

#include <cuda_runtime.h>

namespace lulesh {

namespace {

// A double whose operations round one by one: never contracted.
struct Rounded {
    double v;
    __device__ Rounded() = default;
    __device__ explicit Rounded(double a) : v(a) {}
    friend __device__ Rounded operator+(Rounded a, Rounded b) { return Rounded(__dadd_rn(a.v, b.v)); }
    friend __device__ Rounded operator-(Rounded a, Rounded b) { return Rounded(__dsub_rn(a.v, b.v)); }
    friend __device__ Rounded operator*(Rounded a, Rounded b) { return Rounded(__dmul_rn(a.v, b.v)); }
};

__device__ __forceinline__ double plane_coord(int i, int s)
{
    return i ? __ddiv_rn(__dmul_rn(1.125, (double)i), (double)s) : 0.0;
}

__device__ double cube_volume(int p, int r, int c, int s)
{
    const Rounded x0(plane_coord(c, s)), x1(plane_coord(c + 1, s));
    const Rounded y0(plane_coord(r, s)), y1(plane_coord(r + 1, s));
    const Rounded z0(plane_coord(p, s)), z1(plane_coord(p + 1, s));
    const Rounded x[8] = {x0, x1, x1, x0, x0, x1, x1, x0};
    const Rounded y[8] = {y0, y0, y1, y1, y0, y0, y1, y1};
    const Rounded z[8] = {z0, z0, z0, z0, z1, z1, z1, z1};
    return elem_volume<Rounded>(x, y, z).v;
}

// 1/a of an entity, or with even set of the mean with its mirror image's
// (rows and columns exchanged), which the set-up's sums leave an ulp apart:
// the double-float kernels keep a mirror-symmetric state exactly symmetric
// (dfpack.cuh), and these are the only data that would disturb it.
__device__ __forceinline__ double reciprocal_of(bool even, double a, double image)
{
    return __ddiv_rn(1.0, even ? __dmul_rn(0.5, __dadd_rn(a, image)) : a);
}

// The writable views of a Dom's mesh arrays.
struct MeshOut {
    int *nodelist, *elem_bc;
    unsigned char *node_bc;
    double *volo, *elem_mass, *inv_volo, *nodal_mass, *inv_mass;
    double *x, *y, *z, *e, *v;
    int ne, nn;
    bool even;
};
MeshOut mesh_out(const Dom &d)
{
    return {const_cast<int *>(d.nodelist), const_cast<int *>(d.elem_bc), const_cast<unsigned char *>(d.node_bc),
            const_cast<double *>(d.volo), const_cast<double *>(d.elem_mass), d.inv_volo,
            const_cast<double *>(d.nodal_mass), d.inv_mass, d.x, d.y, d.z, d.e, d.v, d.ne, d.nn,
            d.df == kArithDF64};
}

// The block's cube: a tile belongs to one (tile_cube null: there is only one).
__device__ __forceinline__ CubeDesc cube_of_block(const CubeDesc &one, const CubeDesc *cubes, const int *tile_cube)
{
    return tile_cube ? cubes[tile_cube[blockIdx.x]] : one;
}

__global__ void __launch_bounds__(kTile) k_cube_elements(const __grid_constant__ MeshOut m, const __grid_constant__ CubeDesc one,
                                                         const CubeDesc *cubes, const int *tile_cube)
{
    const int k = blockIdx.x * kTile + threadIdx.x;
    if (k >= m.ne) return;
    const CubeDesc q = cube_of_block(one, cubes, tile_cube);
    const int s = q.s, i = k - q.elem_begin;
    if (i >= s * s * s) {   // a batch's padding: whole-array kernels divide by these
        m.volo[k] = m.elem_mass[k] = m.inv_volo[k] = 1.0;
        return;
    }
    const int c = i % s, r = (i / s) % s, p = i / (s * s);
    const int en = s + 1, n0 = q.node_begin + (p * en + r) * en + c;
    int4 *l = reinterpret_cast<int4 *>(m.nodelist + 8 * (size_t)k);
    l[0] = make_int4(n0, n0 + 1, n0 + en + 1, n0 + en);
    l[1] = make_int4(n0 + en * en, n0 + en * en + 1, n0 + en * en + en + 1, n0 + en * en + en);
    m.elem_bc[k] = (c == 0 ? BC_XI_M_SYMM : 0) | (c == s - 1 ? BC_XI_P_FREE : 0) | (r == 0 ? BC_ETA_M_SYMM : 0) |
                   (r == s - 1 ? BC_ETA_P_FREE : 0) | (p == 0 ? BC_ZETA_M_SYMM : 0) | (p == s - 1 ? BC_ZETA_P_FREE : 0);
    const double vol = cube_volume(p, r, c, s);
    m.volo[k] = vol;
    m.elem_mass[k] = vol;
    m.inv_volo[k] = reciprocal_of(m.even, vol, m.even ? cube_volume(p, c, r, s) : vol);
    m.v[k] = 1.0;
    if (i == 0) m.e[k] = q.e0;
}

// The node's mass: an eighth of each of its elements' volumes, added in the
// order of the elements.
__device__ double cube_node_mass(const double *volo, int p, int r, int c, int s)
{
    double mass = 0.0;
#pragma unroll
    for (int dp = 1; dp >= 0; --dp)
#pragma unroll
        for (int dr = 1; dr >= 0; --dr)
#pragma unroll
            for (int dc = 1; dc >= 0; --dc) {
                const int ep = p - dp, er = r - dr, ec = c - dc;
                if ((unsigned)ep < (unsigned)s && (unsigned)er < (unsigned)s && (unsigned)ec < (unsigned)s)
                    mass = __dadd_rn(mass, __dmul_rn(volo[(ep * s + er) * s + ec], 0.125));
            }
    return mass;
}

__global__ void __launch_bounds__(kTile) k_cube_nodes(const __grid_constant__ MeshOut m, const __grid_constant__ CubeDesc one,
                                                      const CubeDesc *cubes, const int *tile_cube)
{
    const int n = blockIdx.x * kTile + threadIdx.x;
    if (n >= m.nn) return;
    const CubeDesc q = cube_of_block(one, cubes, tile_cube);
    const int s = q.s, en = s + 1, i = n - q.node_begin;
    if (i >= en * en * en) {   // padding
        m.nodal_mass[n] = m.inv_mass[n] = 1.0;
        return;
    }
    const int c = i % en, r = (i / en) % en, p = i / (en * en);
    m.x[n] = plane_coord(c, s);
    m.y[n] = plane_coord(r, s);
    m.z[n] = plane_coord(p, s);
    m.node_bc[n] = (unsigned char)((c == 0 ? 1 : 0) | (r == 0 ? 2 : 0) | (p == 0 ? 4 : 0));
    const double *volo = m.volo + q.elem_begin;
    const double mass = cube_node_mass(volo, p, r, c, s);
    m.nodal_mass[n] = mass;
    m.inv_mass[n] = reciprocal_of(m.even, mass, m.even ? cube_node_mass(volo, p, c, r, s) : mass);
}

void build(const Dom &d, const CubeDesc &one, const CubeDesc *cubes, const int *etile_cube, const int *ntile_cube,
           cudaStream_t st)
{
    const MeshOut m = mesh_out(d);
    k_cube_elements<<<(unsigned)((d.ne + (long)kTile - 1) / kTile), kTile, 0, st>>>(m, one, cubes, etile_cube);
    k_cube_nodes<<<(unsigned)((d.nn + (long)kTile - 1) / kTile), kTile, 0, st>>>(m, one, cubes, ntile_cube);
}

}  // namespace

void launch_build_cube(const Dom &d, const CubeDesc &cube, cudaStream_t st)
{
    build(d, cube, nullptr, nullptr, nullptr, st);
}

void launch_build_cubes(const Dom &d, const CubeDesc *cubes, const int *etile_cube, const int *ntile_cube, cudaStream_t st)
{
    build(d, CubeDesc{}, cubes, etile_cube, ntile_cube, st);
}

}  // namespace lulesh
