// step_df.cu -- the plain path's element geometry and forces in double-float.
//
// In IEEE FP64 the step is bound by GB300's FP64 pipe (2 FMA per SM per clock),
// not by HBM: ~890 FP64 instructions per zone-cycle against ~1.9 kB moved.
// The element geometry (Walsh modes, cross products, volume derivative, node
// normals, volume, face areas, strain rate) and the stress and
// Flanagan-Belytschko hourglass forces are therefore evaluated here as
// double-float pairs on the FP32 pipe (df64.cuh; ~48 significant bits), with
// the same formulas as the FP64 kernels of step_fp64.cu:
//
//   k_elem_force_df      IntegrateStressForElems + CalcHourglassControlForElems
//                        + CalcFBHourglassForceForElems (LULESH-OMP.cc:853-931,
//                        :1233-1558); corner forces stored as pairs
//   k_node_update_df     the corner gather in nodeElemCornerList order, summed
//                        as pairs and joined once in FP64, then the FP64 node
//                        update (:1613-1683)
//   k_elem_kinematics_df CalcKinematicsForElems + CalcLagrangeElements +
//                        CalcMonotonicQGradientsForElems (:1927-2180); keeps
//                        the modes as pairs for the next force kernel
//
// What stays FP64: the nodal state (positions, velocities, their update), the
// element state (the material kernel's arithmetic is in pairs, the energy
// accumulated in FP64: eos_df.cuh), plus the corner-relative differences that
// every geometric quantity starts from: a mode is a signed sum of corner differences, and
// the differences of neighbouring coordinates are exact in FP64, so the
// pairs carry each mode to ~2^-47 of its own size (the FP64 transform of the
// absolute coordinates carries it to 2^-53 of the coordinates).
#include "lulesh_internal.h"
#include "kernels.h"
#include "common.cuh"
#include "dfpack.cuh"
#include "eos_df.cuh"
#include "batch_kernels.cuh"

#include <cuda_runtime.h>

namespace lulesh {

// The modes of one coordinate of an element's corners.
__device__ __forceinline__ ModePacks field_modes(const double *__restrict__ f, const int nl[8])
{
    double c[8];
    gather8(f, nl, c);
    return walsh_packs(corners_of(c));
}

// Geometry cache (Dom::geo): the modes of x, y, z, xd, yd, zd in the pairs
// that the kernels hold them in, three 16-byte planes per field, then the six
// M4.  The cross products are formed again from them: 170 instructions
// against 288 more bytes per element written and read.  The velocity modes
// are worth their 336 bytes: the kinematics kernel has the linear ones in
// hand and completes them in 6 % more time (1196 -> 1268 us at s=192), and
// the force kernel is spared its 24 gathers, 21 FP64 differences and as many
// conversions (1316 -> 1046 us, 1004 now; s=96 172 -> 135, s=47 28.9 -> 23.2).
__device__ __forceinline__ void store_geometry_df(double *geo, size_t ne, int k, int field, const ModePacks &m)
{
    ulonglong2 *g = reinterpret_cast<ulonglong2 *>(geo) + (size_t)(3 * field) * ne + k;
    g[0] = make_ulonglong2(m.m12.hi, m.m12.lo);
    g[ne] = make_ulonglong2(m.m56.hi, m.m56.lo);
    g[2 * ne] = make_ulonglong2(m.m73.hi, m.m73.lo);
    reinterpret_cast<float2 *>(geo + 36 * ne)[field * ne + k] = as_float2(m.m4);
}
__device__ __forceinline__ ModePacks load_geometry_df(const double *geo, size_t ne, int k, int field)
{
    const ulonglong2 *g = reinterpret_cast<const ulonglong2 *>(geo) + (size_t)(3 * field) * ne + k;
    const ulonglong2 a = __ldg(g), b = __ldg(g + ne), c = __ldg(g + 2 * ne);
    return {{a.x, a.y}, {b.x, b.y}, {c.x, c.y}, as_df(__ldg(reinterpret_cast<const float2 *>(geo + 36 * ne) + field * ne + k))};
}

// The modes of the three coordinates as vectors.
struct Modes {
    V2x3n m12, m56;
    V1x3 m3, m4;
};
__device__ __forceinline__ Modes modes_of(const ModePacks &x, const ModePacks &y, const ModePacks &z)
{
    return {both(V2x3{x.m12, y.m12, z.m12}), both(V2x3{x.m56, y.m56, z.m56}),
            {df2_y(x.m73), df2_y(y.m73), df2_y(z.m73)}, {x.m4, y.m4, z.m4}};
}

// The six cross products that the geometry is made of, in pairs: q1 =
// (M4xM5, M4xM6), q2 = (M3xM1, M3xM2), q3 = (M1xM2, M5xM6), and the normal
// generators n1 = M2xM3 + M4xM5, n2 = M3xM1 + M6xM4, n3 = M1xM2 + M5xM6.
struct Crosses {
    V2x3 q1, q2, q3;
    V1x3 n1, n2, n3;
};
__device__ __forceinline__ Crosses crosses_of(const Modes &m)
{
    Crosses c;
    const V2x3 d = first_of(m.m12), e = first_of(m.m56);
    c.q1 = cross2(dup3(m.m4), m.m56);
    c.q2 = cross2(dup3(m.m3), m.m12);
    c.q3 = cross2_even(pack3(half_x(d), half_x(e)), both(pack3(half_y(d), half_y(e))));
    c.n1 = sum1(half_x(c.q1), minus(half_y(c.q2)));
    c.n2 = sum1(half_x(c.q2), minus(half_y(c.q1)));
    c.n3 = sum1(half_x(c.q3), half_y(c.q3));
    return c;
}

// ---------------------------------------------------------------------
// Element force: stress + Flanagan-Belytschko hourglass, as pairs, in the
// space of the Walsh modes
// ---------------------------------------------------------------------
//
// The hourglass shape vectors are hourgam_m(c) = gamma_m(c) - (dV/dx_c . H_m)/V
// (CalcFBHourglassForceForElems, LULESH-OMP.cc:1291-1473), with gamma_m the
// corner signs of modes 4..7, H_m = M4..M7 and 192 dV/dx_c = sum_i s_i(c) W_i
// over the modes 1..6.  Both contractions with them need only sums over
// modes, never over corners.  With U_i the modes of one velocity component,
//   G   = sum_i W_i U_i                        (192 sum_c dV/dx_c u_c)
//   h_m = coefficient (U_m - (H_m/(192 V)) . G)
//   K   = sum_m (H_m/(192 V)) h_m
// and the corner forces are the inverse transform of
//   F_i = h_i - W_i . K  (h_i = 0 for i < 4; no W_7)
// plus the stress forces, which are linear in the corner signs: (p + q)/64
// times the normal generators in F_1..F_3.  60 products per component
// instead of 64 and the 96 that the shape vectors take, and the transforms
// are additions.  Everything runs on pairs of modes (dfpack.cuh).
__device__ __forceinline__ void elem_force_components(const Dom &d, int k, DevScalars *sc, int dim0, int dim1)
{
    const size_t ne = (size_t)d.ne;
    // the element scalars first: their loads are in flight with the geometry's
    const double pk = __ldg(d.p + k), qk = __ldg(d.q + k), vk = __ldg(d.v + k), volok = __ldg(d.volo + k);
    const double ssk = __ldg(d.ss + k), massk = __ldg(d.elem_mass + k);
    int nl[8];
    load_nodelist(d.nodelist, k, nl);
    // the modes: kept by the previous cycle's kinematics kernel, else formed
    // here by the same function (the same bits)
    ModePacks mx, my, mz;
    const bool kept = d.geo && sc->geo_valid;
    if (kept) {
        mx = load_geometry_df(d.geo, ne, k, 0);
        my = load_geometry_df(d.geo, ne, k, 1);
        mz = load_geometry_df(d.geo, ne, k, 2);
    } else {
        mx = field_modes(d.x, nl);
        my = field_modes(d.y, nl);
        mz = field_modes(d.z, nl);
    }
    // the first velocity component's modes, in flight during the geometry
    ModePacks next;
    if (kept) next = load_geometry_df(d.geo, ne, k, 3 + dim0);

    V2x3 W12, W56, W34;
    V1x3 n1, n2, n3;   // normal generators, times (p + q)/64
    {
        const Modes M = modes_of(mx, my, mz);
        const Crosses X = crosses_of(M);
        const V2x3 d12 = first_of(M.m12), d56 = first_of(M.m56);
        const V1x3 c31 = half_x(X.q2), c32 = half_y(X.q2), c12 = half_x(X.q3);
        // only the sign of the Jacobian volume M3.(M1 x M2)/64 is tested
        // (IntegrateStressForElems, LULESH-OMP.cc:853-903)
        if (dot1(M.m3, c12).value().hi <= 0.f) flag_error(sc, ERR_K1_DETERM, k);
        // W_1..3 = 3 (M2xM3) + M4xM5 and so on, W6 = M3xM5 + M4xM2 and -W5 =
        // M3xM6 + M4xM1 in the halves of a pair, W4 = M2xM6 - M1xM5
        auto scaled = [](const V1x3 &v, float s) { return V1x3{df_scale(v.x, s), df_scale(v.y, s), df_scale(v.z, s)}; };
        const V2x3 w65 = cross2_sum(dup3(M.m3), M.m56, dup3(M.m4), swapped(M.m12));
        const V1x3 w4 = cross1_sum(half_y(d12), half_y(d56), minus(half_x(d12)), half_x(d56));
        W12 = pack3(sum1(X.n1, scaled(c32, -2.f)), sum1(X.n2, scaled(c31, 2.f)));
        W34 = pack3(sum1(X.n3, scaled(c12, 2.f)), w4);
        W56 = pack3(minus(half_y(w65)), half_x(w65));
        const df64 w = to_df((1.0 / 64.0) * (pk + qk));
        auto times = [&](const V1x3 &v) { return V1x3{w * v.x, w * v.y, w * v.z}; };
        n1 = times(X.n1);
        n2 = times(X.n2);
        n3 = times(X.n3);
    }
    // CalcHourglassControlForElems (:1503-1558)
    const double determ = volok * vk;
    if (vk <= 0.0) flag_error(sc, ERR_K1_VOLUME, k);
    const double hourg = d.prm.hgcoef;
    const bool hourglass = gt(hourg, 0.0);
    // H_m/(192 V) in pairs (M5, M6), (M4, M7), and the coefficient; the
    // scalar factors are FP64 (a handful of operations)
    V2x3 H56, H47;
    df2n coef;
    {
        const double r = hourglass ? rcbrt_fast(determ) : 0.0;   // determ^(-1/3)
        const df2n vi = df2_both(df2_dup(to_df((r * r * r) * (1.0 / 192.0))));
        H56 = {df2_mul(mx.m56, vi), df2_mul(my.m56, vi), df2_mul(mz.m56, vi)};
        H47 = {df2_mul(df2_pack(mx.m4, df2_x(mx.m73)), vi), df2_mul(df2_pack(my.m4, df2_x(my.m73)), vi),
               df2_mul(df2_pack(mz.m4, df2_x(mz.m73)), vi)};
        coef = df2_both(df2_dup(to_df(-hourg * 0.01 * ssk * massk * r)));
    }

    // One velocity component per iteration, the loop kept rolled (its body
    // is most of the kernel's instructions); each iteration issues the loads
    // of the next component's modes before its own arithmetic.
#pragma unroll 1
    for (int dim = dim0; dim < dim1; ++dim) {
        // (the component is selected, not indexed, so that it stays in
        // registers)
        auto comp = [&](const V1x3 &v) {
            return df64(dim == 0 ? v.x.hi : (dim == 1 ? v.y.hi : v.z.hi), dim == 0 ? v.x.lo : (dim == 1 ? v.y.lo : v.z.lo));
        };
        const df64 y1 = comp(n1), y2 = comp(n2), y3 = comp(n3);
        df2 F12, F56;
        df64 F3, F4, F7;
        if (hourglass) {
            ModePacks u = next;
            if (!kept) u = field_modes(dim == 0 ? d.xd : (dim == 1 ? d.yd : d.zd), nl);
            else if (dim + 1 < dim1) next = load_geometry_df(d.geo, ne, k, 4 + dim);
            const df2n u12 = df2_both(u.m12), u56 = df2_both(u.m56), u34 = df2_both(df2_pack(df2_y(u.m73), u.m4));
            auto modes_dot = [&](df2 a, df2 b, df2 c) {
                return df2_both(df2_dup(joined(Dot2(a, u12).add(b, u56)).plus(joined(Dot2(c, u34))).value()));
            };
            const df2n Gx = modes_dot(W12.x, W56.x, W34.x);
            const df2n Gy = modes_dot(W12.y, W56.y, W34.y);
            const df2n Gz = modes_dot(W12.z, W56.z, W34.z);
            // v.g - c
            auto excess = [](df2 c, const V2x3 &v, const df2n &gx, const df2n &gy, const df2n &gz) {
                return Dot2(v.x, gx).add(v.y, gy).add(v.z, gz).minus(c);
            };
            const df2 h56 = df2_mul(excess(u.m56, H56, Gx, Gy, Gz).negative(), coef);
            const df2 h47 = df2_mul(excess(df2_pack(u.m4, df2_x(u.m73)), H47, Gx, Gy, Gz).negative(), coef);
            const df2n h56n = df2_both(h56), h47n = df2_both(h47);
            auto shape_dot = [&](df2 a, df2 b) {
                return df2_both(df2_dup(joined(Dot2(a, h56n)).plus(joined(Dot2(b, h47n))).value()));
            };
            const df2n Kx = shape_dot(H56.x, H47.x), Ky = shape_dot(H56.y, H47.y), Kz = shape_dot(H56.z, H47.z);
            F12 = excess(df2_pack(y1, y2), W12, Kx, Ky, Kz).raw_negative();
            F56 = excess(h56, W56, Kx, Ky, Kz).raw_negative();
            const df2 F34 = excess(df2_pack(y3, df2_x(h47)), W34, Kx, Ky, Kz).raw_negative();
            F3 = df2_x(F34);
            F4 = df2_y(F34);
            F7 = df2_y(h47);
        } else {
            const df64 zero(0.f, 0.f);
            F12 = df2_pack(y1, y2);
            F56 = df2_pack(zero, zero);
            F3 = y3;
            F4 = F7 = zero;
        }
        df2 f[4];
        inverse_walsh_packs(F12, F56, F3, F4, F7, f);
        float2 *out = reinterpret_cast<float2 *>(dim == 0 ? d.fcx : (dim == 1 ? d.fcy : d.fcz)) + k;
        const int corner[4][2] = {{2, 1}, {0, 3}, {6, 5}, {4, 7}};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            out[corner[c][0] * ne] = as_float2(df2_x(f[c]));
            out[corner[c][1] * ne] = as_float2(df2_y(f[c]));
        }
    }
}

__device__ __forceinline__ void elem_force_df(const Dom &d, int k, DevScalars *sc) { elem_force_components(d, k, sc, 0, 3); }

// 168 registers, three blocks of 128 threads per SM: the FP32 pipe is 71 %
// busy, the rest dependent results.  1004 us at s=192 in mid-blast, 970 from
// the Sedov start (in mid-blast 1850 in scalar pairs over the corners, 1316 on
// packed pairs over the modes, then the velocities' modes kept); when it was
// 1024, four blocks at 128 registers took 1090, blocks of 64 threads 1036, of
// 192 1105, of 384 1301.
__global__ void __launch_bounds__(kBlockElem) k_elem_force_df(const __grid_constant__ Dom d)
{
    if (skip_step(d)) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.ne) return;
    elem_force_df(d, k, d.sc);
}

// Meshes that leave most of the SMs' warp slots empty run one thread per
// element and component (blockIdx.y): the geometry is formed three times, but
// a thread's chain is little more than half as long, and its length is what
// the kernel takes there.  A cycle at s=10 27.9 us against 29.1 in one thread
// per element, s=22 30.6 and 31.5, s=24 the same, s=30 34.6 and 33.3.  (The
// kinematics kernel in three parts, which would convert the positions three
// times, gains nothing: 28.5 at s=10 and 32.7 against 30.4 at s=19.)
constexpr int kByComponentElems = 12000;
__global__ void __launch_bounds__(kBlockElem) k_elem_force_df_by_component(const __grid_constant__ Dom d)
{
    if (skip_step(d)) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.ne) return;
    elem_force_components(d, k, d.sc, blockIdx.y, blockIdx.y + 1);
}

// ---------------------------------------------------------------------
// Node update: the corner gather as pairs, joined once in FP64
// ---------------------------------------------------------------------
//
// On the structured cube the sum is a tree: in each plane of elements the
// two on the diagonal and the two off it, so that exchanging rows and columns
// exchanges operands only and the mirror symmetry that the element kernels
// keep (dfpack.cuh) is not lost here.
__device__ __forceinline__ df64 corner_tree(const df64 f[8])
{
    // list order: (1,1,1) (1,1,0) (1,0,1) (1,0,0) (0,1,1) ... of (dp, dr, dc)
    return ((f[0] + f[3]) + (f[1] + f[2])) + ((f[4] + f[7]) + (f[5] + f[6]));
}
template <bool kEarly>
__device__ __forceinline__ void node_update_df(const Dom &d, int n, const DevScalars *sc)
{
    const float2 *const fc[3] = {reinterpret_cast<const float2 *>(d.fcx), reinterpret_cast<const float2 *>(d.fcy),
                                 reinterpret_cast<const float2 *>(d.fcz)};
    const NodeState state = load_node(d, n);
    df64 f[3] = {df64(0.f, 0.f), df64(0.f, 0.f), df64(0.f, 0.f)};
    const int s = d.s > 0 ? d.s : sc->edge;
    if (kEarly) {
        const CornerSlots at = corner_slots(d, sc, n);
        float2 c[3][8];
        load_corners(at, fc[0], fc[1], fc[2], c);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            df64 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = as_df(c[i][j]);
            if (s > 0) {
                f[i] = corner_tree(v);
            } else {
                f[i] = v[0];
#pragma unroll
                for (int j = 1; j < 8; ++j)
                    if ((at.present >> j) & 1) f[i] = f[i] + v[j];
                for (int j = at.rest; j < at.end; ++j) f[i] = f[i] + as_df(fc[i][__ldg(d.corner_list + j)]);
            }
        }
    } else if (s > 0) {
        const NodePlace at = node_place(d, sc, s, n);
        const size_t ne = (size_t)d.ne;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            auto corner = [&](int dp, int dr, int dc) {
                return at.inside(s, dp, dr, dc) ? as_df(fc[i][corner_of(dp, dr, dc) * ne + at.element(s, dp, dr, dc)])
                                                : df64(0.f, 0.f);
            };
            auto plane = [&](int dp) { return (corner(dp, 1, 1) + corner(dp, 0, 0)) + (corner(dp, 1, 0) + corner(dp, 0, 1)); };
            f[i] = plane(1) + plane(0);
        }
    } else {
        for_listed_corners(d, n, [&](int c, bool first) {
#pragma unroll
            for (int i = 0; i < 3; ++i) f[i] = first ? as_df(fc[i][c]) : f[i] + as_df(fc[i][c]);
        });
    }
    node_integrate(d, n, sc, state, to_double(f[0]), to_double(f[1]), to_double(f[2]));
}

// Twelve blocks per SM (40 registers, 24 bytes spilled): the gather waits on
// memory, and the early loads of load_node (0.387 -> 0.379 ms at s=192) cost
// registers that the compiler would otherwise take 54 of; 0.355 ms at the
// cap, 0.380 at 32 registers.
template <bool kEarly>
__global__ void __launch_bounds__(kBlockNode, kEarly ? 4 : 12) k_node_update_df(const __grid_constant__ Dom d)
{
    if (skip_step(d)) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= d.nn) return;
    if (n == 0 && d.geo) d.sc->geo_valid = 0;   // the positions move: the geometry cache goes stale
    node_update_df<kEarly>(d, n, d.sc);
}

// ---------------------------------------------------------------------
// Element kinematics + monotonic-Q gradients, as pairs
// ---------------------------------------------------------------------

// 64 x the larger |u x v|^2 of the two faces of one direction (hexmodes.cuh):
// |X + Y|^2 and |X - Y|^2 in the halves of a pair.
__device__ __forceinline__ df64 face_pair_max(const V1x3 &X, const V1x3 &Y)
{
    auto comp = [](df64 x, df64 y) {
        const df2 z = df2_add(df2_dup(x), df2_pack(y, -y));
        const f2 h = f2_add(z.hi, z.lo);
        return df2{h, f2_sub(z.lo, f2_sub(h, z.hi))};
    };
    const df2 x = comp(X.x, Y.x), y = comp(X.y, Y.y), z = comp(X.z, Y.z);
    const V2x3 v{x, y, z};
    const df2 n = dot2(v, both(v)).value();
    return fmax(df2_x(n), df2_y(n));
}

__device__ __forceinline__ void elem_kinematics_df(const Dom &d, int k, DevScalars *sc)
{
    const size_t ne = (size_t)d.ne;
    int nl[8];
    load_nodelist(d.nodelist, k, nl);
    const ModePacks mx = field_modes(d.x, nl), my = field_modes(d.y, nl), mz = field_modes(d.z, nl);
    // the next cycle's force kernel works on these same positions and
    // velocities; every context that runs this kernel keeps the cache
    store_geometry_df(d.geo, ne, k, 0, mx);
    store_geometry_df(d.geo, ne, k, 1, my);
    store_geometry_df(d.geo, ne, k, 2, mz);
    if (k == sc->elem_begin) sc->geo_valid = 1;

    const Modes M = modes_of(mx, my, mz);
    const Crosses X = crosses_of(M);
    const V2x3 d12 = first_of(M.m12), d56 = first_of(M.m56);

    // CalcKinematicsForElems, volume part (:1950-1964): 64 V = M3.(M1xM2) +
    // (M1.(M4xM5) + M2.(M6xM4) + M3.(M5xM6))/3 (hexmodes.cuh), in the sums
    // that a mirrored element shares (dfpack.cuh)
    const df64 vol64 = [&] {
        const df64 s = difference(dot2(d12, both(X.q1))).plus(dot1(M.m3, half_y(X.q3))).value();
        return Dot1(s, df64(1.0 / 3.0)).plus(dot1(M.m3, half_x(X.q3))).value();
    }();
    // volume / volo, as a product with the reciprocal taken at set-up, in
    // FP64: it is state, and one product costs less than its two conversions
    const double rel = to_double(df_scale(vol64, 1.f / 64.f)) * __ldg(d.inv_volo + k);
    d.vnew[k] = rel;
    d.delv[k] = rel - d.v[k];
    if (rel <= 0.0) flag_error(sc, ERR_K3_VNEW, k);

    // CalcElemCharacteristicLength (:1821-1862): 4V / sqrt(max AreaFace)
    {
        // a = M3xM4, -b = M5xM2, c = M6xM1; Y1 = b - a, Y2 = c + a, Y3 = c + b
        const V2x3 bc = cross2(d56, swapped(M.m12));
        const V1x3 a = cross1(M.m3, M.m4), nb = half_x(bc), c = half_y(bc);
        const df64 f = fmax(fmax(face_pair_max(X.n1, sum1(nb, a)), face_pair_max(X.n2, sum1(c, a))),
                            face_pair_max(X.n3, sum1(c, minus(nb))));
        reinterpret_cast<float2 *>(d.arealg)[k] = as_float2(df_scale(vol64, 0.25f) * df_rsqrt(f));
    }
    V2x3 V12;   // velocity modes (V1, V2) and V3
    V1x3 V3v;
    {
        auto modes = [&](const double *f, int field, df2 &v12, df64 &v3) {
            const ModePacks u = field_modes(f, nl);
            store_geometry_df(d.geo, ne, k, field, u);
            v12 = u.m12;
            v3 = df2_y(u.m73);
        };
        modes(d.xd, 3, V12.x, V3v.x);
        modes(d.yd, 4, V12.y, V3v.y);
        modes(d.zd, 5, V12.z, V3v.z);
    }
    const V2x3n V21 = swapped(both(V12));

    // CalcMonotonicQGradientsForElems (:2034-2180): the logical differences
    // are M/4, so each cross product is (M x M')/16 and each velocity
    // difference Mv/4; volo vnew is the volume.  eta and xi in the halves of
    // a pair (M3xM1, M3xM2), zeta beside them.  Kept as pairs (Dom::delv_xi).
    {
        const df64 ptiny(1.e-36);
        const df64 vol = df_scale(vol64, 1.f / 64.f);
        // (1/16) (1/4) / (vol + ptiny)
        const df64 vscale = df_rcp(df_scale(vol + ptiny, 64.f));
        const df2 nn = dot2(X.q2, both(X.q2)).value();
        const df2 dv = dot2(X.q2, V21).value();
        const V1x3 c12 = half_x(X.q3);
        auto delx = [&](df64 n) { return as_float2(vol * df_rsqrt(df_scale(n, 0.00390625f) + ptiny)); };
        auto at = [&](double *f) { return reinterpret_cast<float2 *>(f) + k; };
        *at(d.delx_eta) = delx(df2_x(nn));
        *at(d.delx_xi) = delx(df2_y(nn));
        *at(d.delx_zeta) = delx(dot1(c12, c12).value());
        *at(d.delv_eta) = as_float2(vscale * df2_x(dv));
        *at(d.delv_xi) = as_float2(vscale * -df2_y(dv));   // M2xM3 = -M3xM2
        *at(d.delv_zeta) = as_float2(vscale * dot1(c12, V3v).value());
    }

    // CalcKinematicsForElems, strain-rate part (:1975-2020): the half-step
    // Jacobian's columns (M - dt/2 V)/8, the rate their cofactors . V over
    // their determinant (strain_rate, hexmodes.cuh); cof = (CxA, CxB)
    {
        const df64 dt2 = to_df(0.5 * sc->deltatime);
        const df2n nd = df2_both(df2_dup(dt2));
        auto back2 = [&](df2 m, df2 v) { return Dot2(v, nd).minus(m).negative(); };
        auto back1 = [&](df64 m, df64 v) { return Dot1(v, -dt2).plus(Dot1(m.hi, m.lo)).value(); };
        const V2x3 AB{back2(d12.x, V12.x), back2(d12.y, V12.y), back2(d12.z, V12.z)};
        const V1x3 C{back1(M.m3.x, V3v.x), back1(M.m3.y, V3v.y), back1(M.m3.z, V3v.z)};
        const V2x3 cof = cross2(dup3(C), both(AB));
        const V1x3 cze = cross1_even(half_x(AB), half_y(AB));
        const df64 num = dot1(cze, V3v).plus(difference(dot2(cof, V21))).value();
        reinterpret_cast<float2 *>(d.vdov)[k] = as_float2(df_div(num, dot1(C, cze).value()));
    }
}

// 128 registers, two blocks of 256 threads per SM (kin_block).  The work is
// spread over the FP32 pipe (52 % busy), the FP64 pipe (43 %: the 42 exact
// corner differences) and the integer pipe (41 %: their conversions); what
// remains is dependent results and the gathers.  1224 us at s=192 (1619 in
// scalar pairs, 1196 on packed pairs, 1268 with the velocities' modes completed
// and kept, less the conversions' second path); blocks of 192 threads, three
// per SM, 1255, two of 288 1289, one of 512 1312.
__global__ void __launch_bounds__(kKinBlockFactor * kBlockElem, 2) k_elem_kinematics_df(const __grid_constant__ Dom d)
{
    if (skip_step(d)) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.ne) return;
    elem_kinematics_df(d, k, d.sc);
}

// ---------------------------------------------------------------------
// Monotonic-Q limiter and viscosity coefficients as pairs, then the FP64
// material update, volume update and constraint candidates
// ---------------------------------------------------------------------

// One direction of the monotonic limiter (LULESH-OMP.cc:2198-2228) as
// pairs.  The neighbour slopes are divided by the element's own (plus
// 1e-36): in FP64 a vanishing own slope makes the ratios huge but finite,
// and the clamp to [0, max_slope] absorbs them; in pairs the product would
// overflow (and its remainder turn into a NaN), so a ratio whose magnitude
// exceeds 2^100 -- judged from the high words before multiplying -- is
// taken as +-2^100.  That changes no outcome: a ratio beyond it is never the
// minimum unless both are, and then the result is max_slope either way; a
// negative one makes the result 0 either way.
// dm, dp: the neighbours' slopes (of any element where the face has a flag).
__device__ __forceinline__ df64 limiter_phi_df(df64 own, df64 dm, df64 dp, int bm, int bp, int m_symm, int p_symm,
                                               df64 limiter, df64 max_slope)
{
    const df64 norm = df_rcp(own + df64(1.e-36));
    const df64 zero(0.f, 0.f);   // beyond a free face
    if (bm != 0) dm = bm == m_symm ? own : zero;
    if (bp != 0) dp = bp == p_symm ? own : zero;
    const float big = 1.2676506e30f;   // 2^100
    auto ratio = [&](df64 a) {
        if (fabsf(a.hi) * fabsf(norm.hi) > big)   // may be inf: still > big
            return (a.hi < 0.f) != (norm.hi < 0.f) ? df64(-big, 0.f) : df64(big, 0.f);
        return a * norm;
    };
    df64 delvm = ratio(dm), delvp = ratio(dp);
    df64 phi = df_scale(delvm + delvp, 0.5f);
    delvm = delvm * limiter;
    delvp = delvp * limiter;
    if (df_gt(phi, delvm)) phi = delvm;
    if (df_gt(phi, delvp)) phi = delvp;
    if (phi.hi < 0.f) phi = df64(0.f, 0.f);
    if (df_gt(phi, max_slope)) phi = max_slope;
    return phi;
}

// Monotonic-Q region (:2182-2320) and the material update as pairs (the
// energy accumulated in FP64), and the element's constraint keys in pairs
// when kConstraints.
template <bool kConstraints>
__device__ __forceinline__ void elem_material_df(const Dom &d, int k, DevScalars *sc, unsigned long long &kc,
                                                 unsigned long long &kh)
{
    const int bc = __ldg(d.elem_bc + k);
    const MaterialIn in = load_material(d, k);
    const double vnew = d.vnew[k], mass = __ldg(d.elem_mass + k), volo = __ldg(d.volo + k);
    auto pairs = [](const double *f) { return reinterpret_cast<const float2 *>(f); };
    const df64 vdov = as_df(pairs(d.vdov)[k]), arealg = as_df(pairs(d.arealg)[k]);
    const FaceNeighbours nb = face_neighbours(d, sc, k);
    const df64 lim = as_df(d.pairs.limiter_mult), maxs = as_df(d.pairs.max_slope);
    const float2 *dv_xi = pairs(d.delv_xi), *dv_eta = pairs(d.delv_eta), *dv_zeta = pairs(d.delv_zeta);
    const df64 own_xi = as_df(dv_xi[k]), own_eta = as_df(dv_eta[k]), own_zeta = as_df(dv_zeta[k]);
    // the neighbours' slopes without waiting for the face flags: where a flag
    // replaces one, whatever element its clamped index names is loaded
    auto near_k = [&](const float2 *f, int i) { return as_df(f[min(max(i, 0), d.ne - 1)]); };
    const df64 xm = near_k(dv_xi, nb.xim), xp = near_k(dv_xi, nb.xip), em = near_k(dv_eta, nb.etam);
    const df64 ep = near_k(dv_eta, nb.etap), zm = near_k(dv_zeta, nb.zetam), zp = near_k(dv_zeta, nb.zetap);
    const df64 phixi = limiter_phi_df(own_xi, xm, xp, bc & BC_XI_M, bc & BC_XI_P, BC_XI_M_SYMM, BC_XI_P_SYMM, lim, maxs);
    const df64 phieta = limiter_phi_df(own_eta, em, ep, bc & BC_ETA_M, bc & BC_ETA_P, BC_ETA_M_SYMM, BC_ETA_P_SYMM, lim, maxs);
    const df64 phizeta = limiter_phi_df(own_zeta, zm, zp, bc & BC_ZETA_M, bc & BC_ZETA_P, BC_ZETA_M_SYMM, BC_ZETA_P_SYMM,
                                        lim, maxs);
    df64 qlin(0.f, 0.f), qquad(0.f, 0.f);
    if (!(vdov.hi > 0.f)) {
        // the products delv * delx; a positive one contributes nothing
        auto prod = [](df64 dv, df64 dx) {
            const df64 p = dv * dx;
            return p.hi > 0.f ? df64(0.f, 0.f) : p;
        };
        const df64 dxi = prod(own_xi, as_df(pairs(d.delx_xi)[k]));
        const df64 deta = prod(own_eta, as_df(pairs(d.delx_eta)[k]));
        const df64 dzeta = prod(own_zeta, as_df(pairs(d.delx_zeta)[k]));
        const df64 rho = df_div(to_df(mass), to_df(volo) * to_df(vnew));
        const df64 one(1.f, 0.f);
        const df64 lin = (dxi * (one - phixi) + deta * (one - phieta)) + dzeta * (one - phizeta);
        const df64 quad = (dxi * dxi * (one - phixi * phixi) + deta * deta * (one - phieta * phieta)) +
                          dzeta * dzeta * (one - phizeta * phizeta);
        qlin = -(as_df(d.pairs.qlc_monoq) * rho) * lin;
        qquad = as_df(d.pairs.qqc_monoq) * rho * quad;
    }
    if (d.keep & 2) {
        d.ql[k] = to_double(qlin);
        d.qq[k] = to_double(qquad);
    }
    const double ssn = material_update_df<SeriesFn>(d, k, sc, in, vnew, qlin, qquad, d.reps ? __ldg(d.reps + k) : 1);
    if (kConstraints)
        constraint_keys_df<SeriesFn>(to_df(ssn), vdov, arealg, vdov.hi != 0.f, vdov.hi < 0.f, d.pairs, kc, kh);
}

// 32 warps per SM (64 registers, ~40 bytes spilled; 80 registers at 24): the
// kernel waits on its neighbour loads, and the extra warps hide them better
// than the spills cost (0.88 ms at 24 warps, 0.81 at 28, 0.78 at 32, s=192,
// when it took that long).  With cheaper conversions and the parameters'
// pairs from the host it took 0.48 ms, 0.50 with the functions' second word.
template <bool kConstraints>
__global__ void __launch_bounds__(kMatBlockFactor * kBlockElem, 2) k_elem_material_df(const __grid_constant__ Dom d)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long kc = ~0ULL, kh = ~0ULL;
    if (t < d.ne && !skip_step(d)) {
        // with regions, threads take elements in cost-grouped order
        const int k = d.mat_order ? __ldg(d.mat_order + t) : t;
        elem_material_df<kConstraints>(d, k, d.sc, kc, kh);
    }
    if (kConstraints) block_min_publish(kc, kh, d.sc);
}

// ---------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------
static inline unsigned blocks_for(long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

void launch_elem_force_df(const Dom &d, cudaStream_t st)
{
    const unsigned grid = blocks_for(d.ne, elem_block(d));
    if (d.ne < kByComponentElems) k_elem_force_df_by_component<<<dim3(grid, 3), elem_block(d), 0, st>>>(d);
    else k_elem_force_df<<<grid, elem_block(d), 0, st>>>(d);
}

void launch_node_update_df(const Dom &d, cudaStream_t st)
{
    const unsigned grid = blocks_for(d.nn, node_block(d));
    if (d.nn < kEarlyNodes) k_node_update_df<true><<<grid, node_block(d), 0, st>>>(d);
    else k_node_update_df<false><<<grid, node_block(d), 0, st>>>(d);
}

void launch_elem_kinematics_df(const Dom &d, cudaStream_t st)
{
    k_elem_kinematics_df<<<blocks_for(d.ne, kin_block(d)), kin_block(d), 0, st>>>(d);
}

void launch_elem_material_df(const Dom &d, cudaStream_t st, const CycleEnd *end)
{
    if (end) k_elem_material_df<true><<<blocks_for(d.ne, mat_block(d)), mat_block(d), 0, st>>>(d);
    else k_elem_material_df<false><<<blocks_for(d.ne, mat_block(d)), mat_block(d), 0, st>>>(d);
}

// Batched ensembles: kernels 0..3 (force, node update, kinematics, material)
// over the active tiles of one class.
void launch_batch_kernel_df(const Dom &d, const BatchView &b, cudaStream_t st, int kernel, int cls, LaunchCfg cfg)
{
    switch (kernel) {
    case 0: kb_elem<elem_force_df, 168><<<cfg.grid, cfg.block, 0, st>>>(d, b, cls); break;
    case 1:
        if (d.nn < kEarlyNodes) kb_node<node_update_df<true>, 128><<<cfg.grid, cfg.block, 0, st>>>(d, b, cls);
        else kb_node<node_update_df<false>, 64><<<cfg.grid, cfg.block, 0, st>>>(d, b, cls);
        break;
    case 2: kb_elem<elem_kinematics_df, 128><<<cfg.grid, cfg.block, 0, st>>>(d, b, cls); break;
    default: kb_material_capped<elem_material_df<true>, 4><<<cfg.grid, cfg.block, 0, st>>>(d, b, cls); break;
    }
}

int batch_max_blocks_df(int kernel, int block, bool early)
{
    int n = 0;
    cudaError_t e;
    switch (kernel) {
    case 0: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_elem<elem_force_df, 168>, block, 0); break;
    case 1:
        e = early ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_node<node_update_df<true>, 128>, block, 0)
                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_node<node_update_df<false>, 64>, block, 0);
        break;
    case 2: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_elem<elem_kinematics_df, 128>, block, 0); break;
    default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kb_material_capped<elem_material_df<true>, 4>, block, 0); break;
    }
    return e == cudaSuccess ? n : 0;
}

// ---------------------------------------------------------------------
// Pair fields for the host.  On the device, beside the copy: a loop over the
// field on the host took 70 us of get_field's 89 at 104k elements, 650 of
// 711 at a million.
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pairs_to_doubles(const float2 *__restrict__ in, double *__restrict__ out, long n)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 w = in[i];
    out[i] = (double)w.x + (double)w.y;
}
__global__ void __launch_bounds__(256) k_doubles_to_pairs(const double *__restrict__ in, float2 *__restrict__ out, long n)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = in[i];
    float hi = __double2float_rn(a);
    // a strain rate below the floats' range still moves (constraint_keys_df)
    if (hi == 0.f && a != 0.0) hi = copysignf(__uint_as_float(1u), hi);
    out[i] = make_float2(hi, isfinite(hi) ? __double2float_rn(a - (double)hi) : 0.f);
}
void launch_pairs_to_doubles(const double *pairs, double *out, long n, cudaStream_t st)
{
    k_pairs_to_doubles<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float2 *>(pairs), out, n);
}
void launch_doubles_to_pairs(const double *in, double *pairs, long n, cudaStream_t st)
{
    k_doubles_to_pairs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, reinterpret_cast<float2 *>(pairs), n);
}

// ---------------------------------------------------------------------
// Accuracy of the pairs' reciprocal, quotient and roots: squared relative
// errors summed into sums[0..7] and the largest (as bit patterns) in
// worst[0..7], 1/b, a/b, 1/sqrt(a), sqrt(a) by SeriesFn, then by NewtonFn,
// over n pairs spread over [2^-40, 2^40).  A pair's sum fits a double but for
// a rounding of 2^-53, so the defining equation in FP64, each product's
// remainder included, gives its error to that.
// ---------------------------------------------------------------------
__device__ __forceinline__ unsigned long long mixed(unsigned long long z)   // Steele, Lea and Flood's splitmix64
{
    z += 0x9e3779b97f4a7c15ULL;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}
template <class Fn>
__device__ void pair_errors(df64 a, df64 b, double err[4])
{
    auto sum = [](df64 v) { return (double)v.hi + (double)v.lo; };
    const double x = sum(a), y = sum(b);
    const double rcp = sum(Fn::rcp(b)), quot = sum(Fn::div(a, b)), irt = sum(Fn::rsqrt(a)), root = sum(Fn::sqrt(a));
    const double sq = irt * irt, sq_rest = fma(irt, irt, -sq);
    err[0] = fma(y, rcp, -1.0);
    err[1] = fma(y, quot, -x) / x;
    err[2] = 0.5 * fma(sq_rest, x, fma(sq, x, -1.0));
    err[3] = 0.5 * fma(root, root, -x) / x;
}
__global__ void __launch_bounds__(256) k_pair_probe(double *sums, unsigned long long *worst, int n)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    auto value = [&](unsigned long long k) {
        const unsigned long long r = mixed(2ULL * i + k);
        return to_df(ldexp(1.0 + (double)(r >> 11) * 0x1p-53, (int)(mixed(r) % 80) - 40));
    };
    const df64 a = value(0), b = value(1);
    double err[8];
    pair_errors<SeriesFn>(a, b, err);
    pair_errors<NewtonFn>(a, b, err + 4);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        atomicAdd(sums + j, err[j] * err[j]);
        atomicMax(worst + j, (unsigned long long)__double_as_longlong(::fabs(err[j])));
    }
}
void launch_pair_probe(double *sums, unsigned long long *worst, int n, cudaStream_t st)
{
    k_pair_probe<<<(n + 255) / 256, 256, 0, st>>>(sums, worst, n);
}

}  // namespace lulesh
