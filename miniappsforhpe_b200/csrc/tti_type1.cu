// Type1 discretisation of the TTI p/q system (kernels/kernel_type1_gpu_*.cu):
// constant density, centred second derivatives (DF2 least-squares
// coefficients, kernels/fd_coef.h:516-521) on the normal directions and the
// same diagonal form for the mixed ones, applied directly to p and q with no
// first-derivative stage.  Drop-in launchers for the reference's three type1
// entry points:
//   fwd_main_loop_2_1_inner_gpu::launch  (kernel_type1_gpu_fwd.h:6-9)
//   adj_main_loop_2_inner_gpu::launch    (kernel_type1_gpu_adj.h:6-9)
//   launch_update_grad_loop_kernel       (kernel_type1_gpu_grad.h:4-7)
// One thread per cell forward; the adjoint first forms the point-wise transposed
// model (lap/hz of both fields) in the library's four-float scratch, then
// marches through it.  The arithmetic follows the launchers' default
// (optimised) kernels: the derivative sums of compute_z_contributions /
// compute_xy_contributions (kernel_type1_gpu_fwd.cu:150-232,
// kernel_type1_gpu_adj.cu:162-217) and the V/H combination of
// compute_result (kernel_type1_gpu_fwd.cu:122-146).
#include <cuda_runtime.h>

#include <cstdint>

#include "tti_common.cuh"
#include "tti_internal.cuh"
#include "tti_march.cuh"

namespace tti {
namespace {

constexpr int T1X = 32, T1Y = 8;

struct R6 {
    int ixbeg, ixend, iybeg, iyend, izbeg, izend;
};

inline dim3 t1_grid(const R6& r)
{
    return dim3((r.ixend - r.ixbeg + T1X) / T1X, (r.iyend - r.iybeg + T1Y) / T1Y, r.izend - r.izbeg + 1);
}

struct FdConst {
    float xx, yy, zz, xy, yz, zx;
};

// kernel_utils::compute_fd_const (kernels/kernel_utils.h:89-101)
FdConst fd_const(double dx, double dy, double dz)
{
    return FdConst{(float)(1.0 / (dx * dx)), (float)(1.0 / (dy * dy)), (float)(1.0 / (dz * dz)),
                   (float)(1.0 / (4 * dx * dy)), (float)(1.0 / (4 * dy * dz)), (float)(1.0 / (4 * dx * dz))};
}

struct Drv {
    float xx, yy, zz, xy, yz, zx;
};

__device__ __forceinline__ Drv centred(const float* __restrict__ f, int64_t i, int64_t sy, int64_t sz, FdConst k)
{
    float zz = 0.0f, zx = 0.0f, yz = 0.0f;
#pragma unroll
    for (int ir = -4; ir <= 4; ++ir) {
        const float c = c2(ir < 0 ? -ir : ir);
        const int64_t j = i + ir * sz;
        zz = zz + c * __ldg(f + j);
        if (ir != 0) {
            zx = zx + c * (__ldg(f + j + ir) - __ldg(f + j - ir));
            yz = yz + c * (__ldg(f + j + ir * sy) - __ldg(f + j - ir * sy));
        }
    }
    const float f0 = __ldg(f + i);
    float xx = c2(0) * f0, yy = c2(0) * f0, xy = 0.0f;
#pragma unroll
    for (int q = 1; q <= 4; ++q) {
        const float c = c2(q);
        xx += c * (__ldg(f + i + q) + __ldg(f + i - q));
        yy += c * (__ldg(f + i + q * sy) + __ldg(f + i - q * sy));
        xy += c * (__ldg(f + i + q * sy + q) - __ldg(f + i + q * sy - q) + __ldg(f + i - q * sy - q) -
                   __ldg(f + i - q * sy + q));
    }
    return Drv{xx * k.xx, yy * k.yy, zz * k.zz, xy * k.xy, yz * k.yz, zx * k.zx};
}

// MODE 0: f3,f4 += rhs*dt;  1: f = A f + B rhs dt (sponge);  2: rhs into
// halo-free outputs (calc_snap).
template <int MODE>
__global__ void __launch_bounds__(T1X* T1Y)
    k_t1_fwd(float* __restrict__ f3, float* __restrict__ f4, const float* __restrict__ f1,
             const float* __restrict__ f2, const float* __restrict__ m1, const float* __restrict__ m2,
             const float* __restrict__ m3, const float* __restrict__ m4, const float* __restrict__ m5,
             const float* __restrict__ m6, const float* __restrict__ m7, const float2* __restrict__ abx,
             const float2* __restrict__ aby, const float2* __restrict__ abz, R6 r, int ldimx, int ldimy, int ldox,
             int ldoy, float dt, FdConst k)
{
    const int ix = r.ixbeg + blockIdx.x * T1X + threadIdx.x;
    const int iy = r.iybeg + blockIdx.y * T1Y + threadIdx.y;
    const int iz = r.izbeg + blockIdx.z;
    if (ix > r.ixend || iy > r.iyend) return;
    const int64_t sy = ldimx, sz = (int64_t)ldimx * ldimy;
    const int64_t i = iz * sz + (int64_t)iy * sy + ix;
    const Drv a = centred(f1, i, sy, sz, k);
    const Drv b = centred(f2, i, sy, sz, k);
    const float rx = __ldg(m5 + i), ry = __ldg(m6 + i), rz = __ldg(m7 + i);
    const float rxx = rx * rx, ryy = ry * ry, rzz = rz * rz;
    const float rxy = 2.0f * rx * ry, ryz = 2.0f * ry * rz, rzx = 2.0f * rz * rx;
    const float V1 = rxx * a.xx + ryy * a.yy + rzz * a.zz + rxy * a.xy + rzx * a.zx + ryz * a.yz;
    const float H1 = a.xx + a.yy + a.zz - V1;
    const float V2 = rxx * b.xx + ryy * b.yy + rzz * b.zz + rxy * b.xy + rzx * b.zx + ryz * b.yz;
    const float H2 = b.xx + b.yy + b.zz - V2;
    const float r3 = __ldg(m1 + i) * H1 + __ldg(m4 + i) * V1 + __ldg(m2 + i) * V2;
    const float r4 = __ldg(m2 + i) * H1 + __ldg(m3 + i) * V2 + __ldg(m4 + i) * H2;
    if constexpr (MODE == 2) {
        const int64_t o = ((int64_t)(iz - r.izbeg) * ldoy + (iy - r.iybeg)) * ldox + (ix - r.ixbeg);
        f3[o] = r3;
        f4[o] = r4;
    } else {
        // output base offset with the input dimensions, then the output strides
        // (kernel_type1_gpu_fwd.cu:488-492 and :283)
        const int64_t o = ((int64_t)r.izbeg * ldimy + r.iybeg) * ldimx +
                          ((int64_t)(iz - r.izbeg) * ldoy + (iy - r.iybeg)) * ldox + ix;
        if constexpr (MODE == 1) {
            const float A = fminf(abx[ix].x, fminf(aby[iy].x, abz[iz].x));
            const float B = fminf(abx[ix].y, fminf(aby[iy].y, abz[iz].y));
            f3[o] = A * f3[o] + B * r3 * dt;
            f4[o] = A * f4[o] + B * r4 * dt;
        } else {
            f3[o] += r3 * dt;
            f4[o] += r4 * dt;
        }
    }
}

// The adjoint: marching (tti_march.cuh), the z, yz and zx terms of each plane
// scattered into a register queue of the outputs L-4 .. L+4, the in-plane terms
// kept beside it and added last, as the reference does.  Bound by latency (16
// warps per SM, issue slots 0.34, waiting on the plane loaded ahead, the shared-
// memory queue and the barriers; HBM 0.14).  150x141x133: 233 us with a form of
// the temporaries per tap, 132 us.
template <bool SPONGE>
__global__ void __launch_bounds__(MNT, 1)
    k_t1_adj(float* __restrict__ f3, float* __restrict__ f4, MarchArgs a, const float2* __restrict__ abx,
             const float2* __restrict__ aby, const float2* __restrict__ abz, float dt, FdConst k)
{
    __shared__ MarchTiles T;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * MX + tx;
    const int x0 = a.ixbeg + blockIdx.x * MX, y0 = a.iybeg + blockIdx.y * MY;
    const int x = x0 + tx, y = y0 + ty;
    const bool owner = x <= a.ixend && y <= a.iyend;
    const int z0 = a.izbeg + blockIdx.z * a.bz, z1 = min(z0 + a.bz - 1, a.izend);
    const int64_t zs = (int64_t)a.ldimx * a.ldimy;
    const MarchCells cells(a, x0, y0, tid);
    MarchCell v[MPOS];
    march_load<false>(a, cells, (int64_t)(z0 - kRadius) * zs, v);
    float2 sq[9];   // z, yz, zx sums, outputs L-4 .. L+4
    float2 xyq[5];  // in-plane sums, outputs L-4 .. L
#pragma unroll
    for (int j = 0; j < 9; ++j) sq[j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < 5; ++j) xyq[j] = make_float2(0.0f, 0.0f);
    int64_t o = ((int64_t)(z0 - 2 * kRadius) * a.ldimy + y) * a.ldimx + x;  // output plane L-4
    for (int L = z0 - kRadius; L <= z1 + kRadius; ++L, o += zs) {
        const bool inplane = L >= z0 && L <= z1;
        march_form<false>(T, v, tid, inplane);
        __syncthreads();
        if (L < z1 + kRadius) march_load<false>(a, cells, (int64_t)(L + 1) * zs, v);
        const float2 tz = T.zz[ty][tx];
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const int ir = 4 - j;
            const float c = c2(ir < 0 ? -ir : ir);
            float a3 = k.zz * c * tz.x, a4 = k.zz * c * tz.y;
            if (ir != 0) {
                const float2 yp = T.yz[ty + 4 + ir][tx], ym = T.yz[ty + 4 - ir][tx];
                const float2 xp = T.zx[ty][tx + 4 + ir], xm = T.zx[ty][tx + 4 - ir];
                a3 = a3 + k.yz * c * (yp.x - ym.x);
                a4 = a4 + k.yz * c * (yp.y - ym.y);
                a3 = a3 + k.zx * c * (xp.x - xm.x);
                a4 = a4 + k.zx * c * (xp.y - xm.y);
            }
            sq[j].x = sq[j].x + a3;
            sq[j].y = sq[j].y + a4;
        }
        xyq[4] = make_float2(0.0f, 0.0f);
        if (inplane) {
            const float2 cx = T.xx[ty][tx + 4], cy = T.yy[ty + 4][tx];
            float xx3 = c2(0) * cx.x, xx4 = c2(0) * cx.y, yy3 = c2(0) * cy.x, yy4 = c2(0) * cy.y;
            float xy3 = 0.0f, xy4 = 0.0f;
#pragma unroll
            for (int q = 1; q <= 4; ++q) {
                const float c = c2(q);
                const float2 xp = T.xx[ty][tx + 4 + q], xm = T.xx[ty][tx + 4 - q];
                xx3 += c * (xp.x + xm.x);
                xx4 += c * (xp.y + xm.y);
                const float2 yp = T.yy[ty + 4 + q][tx], ym = T.yy[ty + 4 - q][tx];
                yy3 += c * (yp.x + ym.x);
                yy4 += c * (yp.y + ym.y);
                const float2 pp = T.xy[ty + 4 + q][tx + 4 + q], pm = T.xy[ty + 4 + q][tx + 4 - q];
                const float2 mm = T.xy[ty + 4 - q][tx + 4 - q], mp = T.xy[ty + 4 - q][tx + 4 + q];
                xy3 += c * (pp.x - pm.x + mm.x - mp.x);
                xy4 += c * (pp.y - pm.y + mm.y - mp.y);
            }
            xyq[4] = make_float2(k.xx * xx3 + k.yy * yy3 + k.xy * xy3, k.xx * xx4 + k.yy * yy4 + k.xy * xy4);
        }
        if (owner && L - 4 >= z0) {
            const float s3 = sq[0].x + xyq[0].x, s4 = sq[0].y + xyq[0].y;
            if constexpr (SPONGE) {
                const int iz = L - 4;
                const float A = fminf(abx[x].x, fminf(aby[y].x, abz[iz].x));
                const float B = fminf(abx[x].y, fminf(aby[y].y, abz[iz].y));
                f3[o] = A * f3[o] + B * s3 * dt;
                f4[o] = A * f4[o] + B * s4 * dt;
            } else {
                f3[o] += s3 * dt;
                f4[o] += s4 * dt;
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) sq[j] = sq[j + 1];
        sq[8] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < 4; ++j) xyq[j] = xyq[j + 1];
        __syncthreads();  // the tiles are formed anew
    }
}

__global__ void __launch_bounds__(T1X* T1Y)
    k_t1_grad(const float* __restrict__ snap_x, const float* __restrict__ snap_z, float* __restrict__ grad,
              const float* __restrict__ adj_x, const float* __restrict__ adj_z, R6 r, int sldx, int sldy, int ldimx,
              int ldimy)
{
    const int ix = r.ixbeg + blockIdx.x * T1X + threadIdx.x;
    const int iy = r.iybeg + blockIdx.y * T1Y + threadIdx.y;
    const int iz = r.izbeg + blockIdx.z;
    if (ix > r.ixend || iy > r.iyend) return;
    const int64_t d = ((int64_t)(iz - r.izbeg) * sldy + (iy - r.iybeg)) * sldx + (ix - r.ixbeg);
    const int64_t i = ((int64_t)iz * ldimy + iy) * ldimx + ix;
    grad[d] += adj_x[i] * snap_x[d] + adj_z[i] * snap_z[d];
}

inline cudaStream_t S(tti_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

bool t1_ranges_ok(int ixbeg, int ixend, int iybeg, int iyend, int izbeg, int izend, int ldimx, int ldimy, int ldimz)
{
    return ranges_ok(ixbeg, ixend, iybeg, iyend, izbeg, izend, ldimx, ldimy) && ldimz >= izend + 1 + kRadius;
}

} // namespace

int launch_t1_adj_with_base(float* f3, float* f4, const float* f1, const float* f2, const float* m1, const float* m2,
                            const float* m3, const float* m4, const float* rx, const float* ry, const float* rz,
                            const float* abx, const float* aby, const float* abz, float4* base, int ixbeg, int ixend,
                            int iybeg, int iyend, int izbeg, int izend, int ldimx, int ldimy, float dt, double dx,
                            double dy, double dz, int use_sponge, cudaStream_t st)
{
    const int rc =
        launch_base(f1, f2, m1, m2, m3, m4, base, ixbeg, ixend, iybeg, iyend, izbeg, izend, ldimx, ldimy, st);
    if (rc) return rc;
    const MarchArgs m{base,  nullptr, rx,    ry,    rz,    ixbeg, ixend, iybeg,
                      iyend, izbeg,   izend, ldimx, ldimy, march_bz(ixend - ixbeg + 1, iyend - iybeg + 1, izend - izbeg + 1)};
    const FdConst k = fd_const(dx, dy, dz);
    const float2* ax = reinterpret_cast<const float2*>(abx);
    const float2* ay = reinterpret_cast<const float2*>(aby);
    const float2* az = reinterpret_cast<const float2*>(abz);
    if (use_sponge)
        k_t1_adj<true><<<march_grid(m), dim3(MX, MY), 0, st>>>(f3, f4, m, ax, ay, az, dt, k);
    else
        k_t1_adj<false><<<march_grid(m), dim3(MX, MY), 0, st>>>(f3, f4, m, ax, ay, az, dt, k);
    return launch_status();
}

} // namespace tti

using namespace tti;

extern "C" {

int tti_launch_type1_fwd(float* field3, float* field4, const float* field1, const float* field2, const float* model1,
                         const float* model2, const float* model3, const float* model4, const float* model5,
                         const float* model6, const float* model7, const float* ABx, const float* ABy,
                         const float* ABz, int ixbeg, int ixend, int iybeg, int iyend, int izbeg, int izend,
                         int ldimx_in, int ldimy_in, int ldimz_in, int ldimx_out, int ldimy_out, int ldimz_out,
                         float dt, double dx, double dy, double dz, int order, tti_stream_t stream, int calc_snap,
                         int use_sponge, int simple)
{
    (void)simple;
    (void)ldimz_out;
    if (order != 8 || (calc_snap && use_sponge)) return TTI_EINVAL;
    if (!t1_ranges_ok(ixbeg, ixend, iybeg, iyend, izbeg, izend, ldimx_in, ldimy_in, ldimz_in)) return TTI_EINVAL;
    if (!field3 || !field4 || !field1 || !field2 || !model1 || !model2 || !model3 || !model4 || !model5 ||
        !model6 || !model7)
        return TTI_EINVAL;
    if (use_sponge && (!ABx || !ABy || !ABz)) return TTI_EINVAL;
    if (calc_snap ? (ldimx_out < ixend - ixbeg + 1 || ldimy_out < iyend - iybeg + 1)
                  : (ldimx_out < ixend + 1 || ldimy_out < iyend - iybeg + 1))
        return TTI_EINVAL;
    const R6 r{ixbeg, ixend, iybeg, iyend, izbeg, izend};
    const FdConst k = fd_const(dx, dy, dz);
    const float2* ax = reinterpret_cast<const float2*>(ABx);
    const float2* ay = reinterpret_cast<const float2*>(ABy);
    const float2* az = reinterpret_cast<const float2*>(ABz);
    const dim3 g = t1_grid(r), b(T1X, T1Y);
    if (calc_snap)
        k_t1_fwd<2><<<g, b, 0, S(stream)>>>(field3, field4, field1, field2, model1, model2, model3, model4, model5,
                                            model6, model7, ax, ay, az, r, ldimx_in, ldimy_in, ldimx_out, ldimy_out,
                                            dt, k);
    else if (use_sponge)
        k_t1_fwd<1><<<g, b, 0, S(stream)>>>(field3, field4, field1, field2, model1, model2, model3, model4, model5,
                                            model6, model7, ax, ay, az, r, ldimx_in, ldimy_in, ldimx_out, ldimy_out,
                                            dt, k);
    else
        k_t1_fwd<0><<<g, b, 0, S(stream)>>>(field3, field4, field1, field2, model1, model2, model3, model4, model5,
                                            model6, model7, ax, ay, az, r, ldimx_in, ldimy_in, ldimx_out, ldimy_out,
                                            dt, k);
    return launch_status();
}

int tti_launch_type1_adj(float* field3, float* field4, const float* field1, const float* field2, const float* model1,
                         const float* model2, const float* model3, const float* model4, const float* model5,
                         const float* model6, const float* model7, const float* ABx, const float* ABy,
                         const float* ABz, int ixbeg, int ixend, int iybeg, int iyend, int izbeg, int izend,
                         int ldimx, int ldimy, int ldimz, float dt, double dx, double dy, double dz, int order,
                         tti_stream_t stream, int use_sponge, int simple)
{
    (void)simple;
    if (order != 8) return TTI_EINVAL;
    if (!t1_ranges_ok(ixbeg, ixend, iybeg, iyend, izbeg, izend, ldimx, ldimy, ldimz)) return TTI_EINVAL;
    if (!field3 || !field4 || !field1 || !field2 || !model1 || !model2 || !model3 || !model4 || !model5 ||
        !model6 || !model7)
        return TTI_EINVAL;
    if (use_sponge && (!ABx || !ABy || !ABz)) return TTI_EINVAL;
    const size_t nelem = (size_t)ldimx * ldimy * (size_t)(izend + 1 + kRadius);
    cudaStream_t st = S(stream);
    const tti::CallScratch scratch(nelem, st);
    float4* base = scratch.get();
    if (!base) return TTI_ENOMEM;
    return launch_t1_adj_with_base(field3, field4, field1, field2, model1, model2, model3, model4, model5, model6, model7,
                                   ABx, ABy, ABz, base, ixbeg, ixend, iybeg, iyend, izbeg, izend, ldimx, ldimy, dt, dx,
                                   dy, dz, use_sponge, st);
}

int tti_launch_type1_update_grad(const float* snap_x, const float* snap_z, float* grad_Vp, const float* adj_x,
                                 const float* adj_z, int ixbeg, int ixend, int iybeg, int iyend, int izbeg, int izend,
                                 int snap_ldimx, int snap_ldimy, int ldimx, int ldimy, tti_stream_t stream)
{
    if (ixend < ixbeg || iyend < iybeg || izend < izbeg || ixbeg < 0 || iybeg < 0 || izbeg < 0) return TTI_EINVAL;
    if (ldimx < ixend + 1 || ldimy < iyend + 1) return TTI_EINVAL;
    if (snap_ldimx < ixend - ixbeg + 1 || snap_ldimy < iyend - iybeg + 1) return TTI_EINVAL;
    if (!snap_x || !snap_z || !grad_Vp || !adj_x || !adj_z) return TTI_EINVAL;
    const R6 r{ixbeg, ixend, iybeg, iyend, izbeg, izend};
    k_t1_grad<<<t1_grid(r), dim3(T1X, T1Y), 0, S(stream)>>>(snap_x, snap_z, grad_Vp, adj_x, adj_z, r, snap_ldimx,
                                                             snap_ldimy, ldimx, ldimy);
    return launch_status();
}

} // extern "C"
