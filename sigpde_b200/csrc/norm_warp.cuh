// norm_warp.cuh -- robust normalisation, one path a warp: the root-find of norm_wave.cuh with every solve on one warp's
// wavefront (wave.cuh), for calls of more paths than CTAs of norm_kernel work on at a time.
//
// norm_kernel shortens one path's chain of solves with up to 16 warps; it pays for that with CTAs whose warps wait for
// one another, and with a tile of nc x nc increments a CTA.  Where the device has more paths than it can give a CTA, a
// warp a path loses nothing to barriers and keeps less: increments come from a tile in shared memory up to
// kNormWarpTileBytes, else they are formed from the differences (or read from the caller's tensor) as the wavefront
// goes, so the workspace does not grow with nc squared.  The cells are norm_kernel's, bit for bit.
#pragma once

#include "norm_wave.cuh"

namespace sigk {

enum : int { kNormDelta = 0, kNormGiven = 1, kNormTile = 2 };
constexpr size_t kNormWarpTileBytes = 48 * 1024;

// Increments from another source, times f (the root-find solves a path again and again with a new scale).
template <class Src, int RC>
struct ScaledIncs {
    Src src;
    double f;

    __device__ __forceinline__ void stage(int64_t ci0, int64_t ncx, int lane, bool rc_per_row)
    {
        src.stage(ci0, ncx, lane, rc_per_row);
    }
    __device__ __forceinline__ void column(int64_t cj, int lane, double (&c)[RC]) const
    {
        src.column(cj, lane, c);
#pragma unroll
        for (int rc = 0; rc < RC; ++rc) c[rc] *= f;
    }
};

// Increments from a warp's tile in shared memory, tile[cj * pitch + ci].
template <int RC>
struct TileIncs {
    const double *tile;
    int64_t pitch;
    int64_t ci0 = 0, ncx = 0;
    bool rc_per_row = false;

    __device__ __forceinline__ void stage(int64_t ci0_, int64_t ncx_, int, bool rc_per_row_)
    {
        ci0 = ci0_;
        ncx = ncx_;
        rc_per_row = rc_per_row_;
    }
    __device__ __forceinline__ void column(int64_t cj, int, double (&c)[RC]) const
    {
        const double *col = tile + cj * pitch;
#pragma unroll
        for (int rc = 0; rc < RC; ++rc) {
            const int64_t ci = ci0 + (rc_per_row ? rc : 0);
            c[rc] = ci < ncx ? col[ci] : 0.0;
        }
    }
};

template <typename TIN, int R, int O, int MODE>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) norm_warp_kernel(NormParams p)
{
    constexpr int RC = BlockShape<R, O>::RC;
    extern __shared__ __align__(16) double norm_warp_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t gwarp = (int64_t)blockIdx.x * kWarpsPerBlock + wib, nwarps = (int64_t)gridDim.x * kWarpsPerBlock;
    const int nc = p.nc;
    const SolveGeom g = make_geom<R, O>(nc, nc, p.order);
    double *bnd = p.bnd ? p.bnd + gwarp * p.bnd_stride : nullptr;
    double *mem = p.smem_values ? norm_warp_smem + wib * p.smem_values : nullptr; // the tile, or the staged differences

    for (int64_t b = gwarp; b < p.n; b += nwarps) {
        auto root = [&](auto src) {
            ScaledIncs<decltype(src), RC> inc{src, 0.0};
            auto solve = [&](double scale) -> double {
                inc.f = p.fscale * scale;
                return warp_solve<double, R, O, true>(g, inc, bnd);
            };
            double out = 0.0;
            int it = 0;
            normalize_path(p, b, lane == 0, solve, out, it);
            if (lane == 0) {
                if (p.lam) {
                    if (p.in64)
                        reinterpret_cast<double *>(p.lam)[b] = out;
                    else
                        reinterpret_cast<float *>(p.lam)[b] = (float)out;
                }
                if (p.iters) p.iters[b] = it;
            }
        };
        if constexpr (MODE == kNormGiven) {
            GivenIncs<double, TIN, RC> src;
            src.inc = reinterpret_cast<const TIN *>(p.inc) + b * p.is0;
            src.si = p.is1;
            src.sj = p.is2;
            src.fscale = 1.0;
            root(src);
        } else if constexpr (MODE == kNormDelta) {
            DeltaIncs<double, RC> src;
            src.dX = p.dx + b * p.d * nc;
            src.dY = src.dX;
            src.d = p.d;
            src.ncy = nc;
            src.dxs = mem;
            root(src);
        } else {
            const double *dx = p.dx + b * p.d * nc;
            __syncwarp(); // the previous path's solves are done with the tile
            for (int e = lane; e < nc * nc; e += 32) {
                const int cj = e / nc, ci = e - cj * nc;
                double acc = 0.0;
                for (int64_t k = 0; k < p.d; ++k) acc = fma(dx[k * nc + ci], dx[k * nc + cj], acc);
                mem[cj * p.pitch + ci] = acc;
            }
            __syncwarp();
            TileIncs<RC> src;
            src.tile = mem;
            src.pitch = p.pitch;
            root(src);
        }
    }
}

} // namespace sigk
