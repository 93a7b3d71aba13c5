// vd_mg2d.cuh -- one leg of a V(2,2) cycle on one 2-D level in one kernel (included by
// vd_poisson.cu and vd_diffusion.cu).
//
// A level of the 2-D multigrids costs eleven launches a cycle when every half sweep,
// the restriction and the prolongation are kernels of their own, and at 4 us each these
// were most of a solve (512^2 and below).  Here a CTA stages a tile of the level with a
// halo of five cells and takes both smoothing sweeps on it: half sweep s updates the
// cells of its colour up to 4 - s cells outside the tile (each half sweep needs one
// more ring of correct neighbours than it leaves), so the tile's own cells get the
// values that half sweeps over the whole grid give, in the same operations.  Going
// down the kernel then restricts the residual; coming up it starts from the
// prolongated correction and can form the residual's maximum.  The result goes to the
// level's other array (a neighbouring tile still reads the old values).
// 32 x 16 tiles of 256 threads: 2.1 staged and 1.5 smoothed cells per cell.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "vd_kernels.cuh"

namespace vd {

constexpr int kMg2X = 32, kMg2Y = 16, kMg2H = 5, kMg2Threads = 256;
constexpr int kMg2W = kMg2X + 2 * kMg2H, kMg2R = kMg2Y + 2 * kMg2H;  // staged columns, rows

// OP supplies the level's discrete operator:
//   T                     value type
//   n[2]                  cells
//   rhs(c)                right-hand side of cell c = i + n0 j
//   kCoef, coef(d, i, j)  number of staged coefficient arrays (0 or 2) and the lower
//                         face's coefficient of direction d (faces 0 .. n[d])
//   row(i, j, vx0, vx1, vy0, vy1, b..., off, diag)   the operator row from neighbours
//   quot(a, b)            the smoother's quotient
//   prolong(i, j)         the coarse correction at the cell (UP)
//   restrict_to(i, j, s)  stores the averaged residual of coarse cell (i, j) (not UP)
template <class OP, bool UP>
__global__ void __launch_bounds__(kMg2Threads) k_mg2d(const __grid_constant__ OP op,
                                                      const typename OP::T* __restrict__ phi_in,
                                                      typename OP::T* __restrict__ phi_out, double* corr,
                                                      unsigned long long* maxout)
{
    grid_wait();
    using T = typename OP::T;
    constexpr int W = kMg2W, R = kMg2R, H = kMg2H;
    __shared__ T sp[W * R], sr[W * R];
    __shared__ T sb[OP::kCoef ? OP::kCoef * W * R : 1];
    const int n0 = op.n[0], n1 = op.n[1];
    const int x0 = blockIdx.x * kMg2X - H, y0 = blockIdx.y * kMg2Y - H;
    for (int q = threadIdx.x; q < W * R; q += kMg2Threads) {
        const int i = x0 + q % W, j = y0 + q / W;
        const bool in = i >= 0 && i < n0 && j >= 0 && j < n1;
        T p = T(0), r = T(0);
        if (in) {
            const int64_t c = i + (int64_t)n0 * j;
            if (phi_in) p = phi_in[c];
            if (UP) p += op.prolong(i, j);
            r = op.rhs(c);
        }
        sp[q] = p;
        sr[q] = r;
        if (OP::kCoef) {
            sb[q] = i >= 0 && i <= n0 && j >= 0 && j < n1 ? op.coef(0, i, j) : T(0);
            sb[W * R + q] = i >= 0 && i < n0 && j >= 0 && j <= n1 ? op.coef(1, i, j) : T(0);
        }
    }
    __syncthreads();
    auto row = [&](int q, int i, int j, T& off, T& diag) {
        if constexpr (OP::kCoef > 0)
            op.row(i, j, sp[q - 1], sp[q + 1], sp[q - W], sp[q + W], sb[q], sb[q + 1], sb[W * R + q], sb[W * R + q + W],
                   off, diag);
        else
            op.row(i, j, sp[q - 1], sp[q + 1], sp[q - W], sp[q + W], off, diag);
    };
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const int m = 4 - s;                       // rings outside the tile
        const int hw = (kMg2X + 2 * m) / 2, nr = kMg2Y + 2 * m;
        for (int t = threadIdx.x; t < hw * nr; t += kMg2Threads) {
            const int lj = H - m + t / hw, j = y0 + lj;
            // the cell of the colour in the pair (x0 + H - m is even or odd with m)
            const int l0 = H - m + 2 * (t % hw);
            const int li = l0 + ((x0 + l0 + j + s) & 1), i = x0 + li;
            if (i < 0 || i >= n0 || j < 0 || j >= n1) continue;
            const int q = li + W * lj;
            T off, diag;
            row(q, i, j, off, diag);
            sp[q] = op.quot(sr[q] - off, diag);
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < kMg2X * kMg2Y; t += kMg2Threads) {
        const int li = H + t % kMg2X, lj = H + t / kMg2X;
        const int i = x0 + li, j = y0 + lj;
        if (i >= n0 || j >= n1) continue;
        const int64_t c = i + (int64_t)n0 * j;
        const T v = sp[li + W * lj];
        phi_out[c] = v;
        if (UP && corr) corr[c] += (double)v;
    }
    if constexpr (!UP) {
        const int t = threadIdx.x;
        if (t < kMg2X * kMg2Y / 4) {
            const int ci = t % (kMg2X / 2), cj = t / (kMg2X / 2);
            const int i0 = x0 + H + 2 * ci, j0 = y0 + H + 2 * cj;
            if (i0 < n0 && j0 < n1) {
                T s = T(0);
#pragma unroll
                for (int dy = 0; dy < 2; dy++)
#pragma unroll
                    for (int dx = 0; dx < 2; dx++) {
                        const int q = H + 2 * ci + dx + W * (H + 2 * cj + dy);
                        T off, diag;
                        row(q, i0 + dx, j0 + dy, off, diag);
                        s += sr[q] - (off + diag * sp[q]);
                    }
                op.restrict_to(i0 / 2, j0 / 2, s * T(0.25));
            }
        }
    } else if (maxout) {
        double m = 0.0;
        for (int t = threadIdx.x; t < kMg2X * kMg2Y; t += kMg2Threads) {
            const int li = H + t % kMg2X, lj = H + t / kMg2X;
            const int i = x0 + li, j = y0 + lj;
            if (i >= n0 || j >= n1) continue;
            const int q = li + W * lj;
            T off, diag;
            row(q, i, j, off, diag);
            const double r = (double)(sr[q] - (off + diag * sp[q]));
            m = fmax(m, r == r ? fabs(r) : INFINITY);  // a NaN residual counts as the largest
        }
        __shared__ double wmax[kMg2Threads / 32];
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kMg2Threads / 32; w++) m = fmax(m, wmax[w]);
            atomicMax(maxout, (unsigned long long)__double_as_longlong(m));
        }
    }
}

inline dim3 mg2d_grid(const int* n)
{
    return dim3((unsigned)((n[0] + kMg2X - 1) / kMg2X), (unsigned)((n[1] + kMg2Y - 1) / kMg2Y));
}

}  // namespace vd
