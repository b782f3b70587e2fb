// Column-marching form of the launchers that differentiate the transposed-model
// temporaries (type2 adjoint derivatives, type1 adjoint).  A block of 32x16
// threads walks z through a column tile.  The temporaries of a plane are formed
// once per cell of the halo'd tile, in shared memory, instead of once per tap
// and output; the values they are formed from are loaded a plane ahead into
// registers, while the stencils of the plane before run.
#pragma once

#include "tti_common.cuh"
#include "tti_internal.cuh"

namespace tti {

constexpr int MX = 32, MY = 16, MNT = MX * MY;
constexpr int MHW = MX + 2 * kRadius, MHH = MY + 2 * kRadius;  // tile with a halo of 4
constexpr int MPOS = (MHW * MHH + MNT - 1) / MNT;              // its cells per thread

// Temporaries of one plane, both fields of a cell side by side.
struct MarchTiles {
    float2 xx[MY][MHW], zx[MY][MHW];  // rows y0.., columns x0-4..
    float2 yy[MHH][MX], yz[MHH][MX];  // rows y0-4.., columns x0..
    float2 xy[MHH][MHW];
    float2 zz[MY][MX];
};
static_assert(sizeof(MarchTiles) <= 48 * 1024, "static shared memory");

// One cell's inputs: the transposed model (s1, h1, s2, h2), the tilt and, type2
// only, the buoyancy.
struct MarchCell {
    float4 b;
    float ir, rx, ry, rz;
};

struct MarchArgs {
    const float4* base;
    const float *irho, *rx, *ry, *rz;
    int ixbeg, ixend, iybeg, iyend, izbeg, izend, ldimx, ldimy;
    int bz;  // output planes per block
};

// A thread's cells of the halo'd tile: offsets inside a plane, -1 outside the
// range (and its halo), where the temporaries are zero and feed no output.
struct MarchCells {
    int off[MPOS];
    __device__ MarchCells(const MarchArgs& a, int x0, int y0, int tid)
    {
#pragma unroll
        for (int k = 0; k < MPOS; ++k) {
            const int e = tid + k * MNT, x = x0 - kRadius + e % MHW, y = y0 - kRadius + e / MHW;
            off[k] = (e < MHW * MHH && x <= a.ixend + kRadius && y <= a.iyend + kRadius) ? y * a.ldimx + x : -1;
        }
    }
};

template <bool RHO>
__device__ __forceinline__ void march_load(const MarchArgs& a, const MarchCells& m, int64_t plane, MarchCell (&v)[MPOS])
{
#pragma unroll
    for (int k = 0; k < MPOS; ++k) {
        v[k] = MarchCell{make_float4(0.0f, 0.0f, 0.0f, 0.0f), 1.0f, 0.0f, 0.0f, 0.0f};
        if (m.off[k] >= 0) {
            const int64_t i = plane + m.off[k];
            v[k].b = __ldg(a.base + i);
            if (RHO) v[k].ir = __ldg(a.irho + i);
            v[k].rx = __ldg(a.rx + i);
            v[k].ry = __ldg(a.ry + i);
            v[k].rz = __ldg(a.rz + i);
        }
    }
}

// The plane's temporaries (kernel_type2_grad_snap.cu:66-132, kernel_type1_gpu_
// adj.cu:103-153).  inplane: an output plane; the planes around a chunk feed
// zz, yz and zx alone.  MIXED: yz, zx and xy are wanted.
template <bool RHO, bool MIXED = true>
__device__ __forceinline__ void march_form(MarchTiles& t, const MarchCell (&v)[MPOS], int tid, bool inplane)
{
#pragma unroll
    for (int k = 0; k < MPOS; ++k) {
        const int e = tid + k * MNT, r = e / MHW, c = e % MHW;
        if (e >= MHW * MHH) continue;
        const float4 b = v[k].b;
        const float rx = v[k].rx, ry = v[k].ry, rz = v[k].rz;
        const float rho = RHO ? 1.0f / v[k].ir : 1.0f;
        auto norm = [&](float w) {
            const float2 n = make_float2(b.x + w * b.y, b.z + w * b.w);
            return RHO ? make_float2(rho * n.x, rho * n.y) : n;
        };
        auto mixed = [&](float w) { return make_float2(w * b.y, w * b.w); };
        const bool rowb = r >= kRadius && r < kRadius + MY, colb = c >= kRadius && c < kRadius + MX;
        if (rowb) {
            if (inplane) t.xx[r - kRadius][c] = norm(rx * rx);
            if (MIXED) t.zx[r - kRadius][c] = mixed(2.0f * rz * rx);
        }
        if (colb) {
            if (inplane) t.yy[r][c - kRadius] = norm(ry * ry);
            if (MIXED) t.yz[r][c - kRadius] = mixed(2.0f * ry * rz);
        }
        if (MIXED && inplane) t.xy[r][c] = mixed(2.0f * rx * ry);
        if (rowb && colb) t.zz[r - kRadius][c - kRadius] = norm(rz * rz);
    }
}

inline dim3 march_grid(const MarchArgs& a)
{
    return dim3((a.ixend - a.ixbeg + MX) / MX, (a.iyend - a.iybeg + MY) / MY, (a.izend - a.izbeg + a.bz) / a.bz);
}

// Output planes per block: the cut of the columns into n chunks with the least
// work on the last SM, one block resident on each and each chunk paying the
// planes around it, which form and scatter about half of what an output's plane
// does.  Chunks of less than 8 planes only while all blocks fit at once: on
// small grids the SMs are idle otherwise, and a march is as long as its chunk.
// Calls with their temporaries' kernel, 8 planes at least -> as here (a thread
// per cell): 48x40x40 adjoint derivatives 27.7 -> 16.6 us (19.2), density
// gradient 23.0 -> 11.7 (10.1), type1 adjoint 28.4 -> 15.6 (13.5); 64^3 28.7 ->
// 21.3 (37.8), 24.0 -> 16.4 (23.1), 29.5 -> 20.9 (27.8); 20^3, nine planes for
// one of output, 29.2 -> 13.7 (11.5), 26.3 -> 9.3 (9.8), 30.1 -> 12.4 (11.1).
// From 80^3 on the cut is as before.
inline int march_bz(int nx, int ny, int nz)
{
    const int64_t tiles = (int64_t)((nx + MX - 1) / MX) * ((ny + MY - 1) / MY), sms = device_sms();
    int best = nz;
    double least = 1e300;
    for (int n = 1; n <= nz; ++n) {
        const int bz = (nz + n - 1) / n;
        const int64_t blocks = tiles * ((nz + bz - 1) / bz);
        if (n > 1 && n > nz / 8 && blocks > sms) break;
        const double cost = (double)((blocks + sms - 1) / sms) * (bz + 0.5 * 2 * kRadius);
        if (cost < least - 1e-9) {
            least = cost;
            best = bz;
        }
    }
    return best;
}

} // namespace tti
