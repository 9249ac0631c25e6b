// kernels_brick.cuh -- both smoothing sweeps of one leg of the V-cycle on a small level, in one launch.
//
// Down leg: two red-black Gauss-Seidel sweeps from x = 0, then b_coarse = restriction of b - A x.  Up leg:
// x + P e, then two sweeps (with <r64, x> summed on level 0).  The same cycle as v_cycle_recursive
// (src/multigrid/cycle/v_cycle.cu:36-74; red = (i+j+k) even first, gsrb_3d.cu:368-576; residual_3d.cu:378-502;
// restrict_3d.cu:12-53; prolong_3d.cu:520-621) and the same values as the sweeps it replaces up to rounding.
//
// A level of 32^3 or 64^3 cells is small: a launch that streams it once (x-pair sweep, residual) takes
// 4 to 9 us whatever it moves, five of them a level and cycle.  Here a CTA owns a brick of 8 x 8 x BZ
// cells and works on it with a halo of four cells, the reach of two sweeps and a residual, so that
// nothing is exchanged between CTAs: each half-sweep is valid on a region one cell smaller than the last.
// The region's cells are recomputed by up to eight bricks, which costs less than the launches as long as
// the bricks are a few per SM.
//
// Each of the 512 threads owns x-pairs of KP consecutive planes (one red and one black cell a pair).  The six
// weights C_f / D and b dx^2 / D of its cells stay in registers; only x is in shared memory, in rows
// padded so that the 32 lanes (8 pairs x 4 rows, alternating colours) hit different banks.  Any sizes,
// periodic axes included (even counts; a region wider than the grid holds copies of a cell that all get
// the same value).
//
// Measured, one leg: 32^3 FP32 8.8 us (two sweeps and the residual 18 us), 32^3 FP64 7.2, 16^3 FP64 7; bound by the
// latency of the coefficient loads, the four barriers and the launch, not by bytes.  Solves of 160 x 96 x 128
// periodic, FP64: 5.20 -> 3.75 ms with the matrix of kernels_tail.cuh below the bricks.
#pragma once
#include "kernels_mg.cuh"
#include "kernels_pcg.cuh"

namespace mf3d {

constexpr int BK_NT = 512, BK_B = 8, BK_H = 4, BK_R = BK_B + 2 * BK_H; // brick edge in x and y, halo, region edge
template <class T> struct BrickGeom {
    static constexpr int KP = sizeof(T) == 4 ? 4 : 3;   // planes per thread (registers decide)
    static constexpr int RZ = 4 * KP, BZ = RZ - 2 * BK_H; // planes of the region and of the brick
    static constexpr int P = sizeof(T) == 4 ? 24 : 16;  // row pitch of x
};

// T: x and the arithmetic; TB: b; TO: the result of an up leg (the first FP64 level below an FP32 one takes b
// and gives x in FP32)
template <class T, class TC, class TB = T, class TO = T> struct BrickLegArgs {
    LevelOp<TC> L;
    const TB* b;
    const T* x_in; // up leg: the down leg's x
    const T* e_c;  // up leg: the coarse correction, coarse dims ncx, ncy
    int ncx, ncy;
    TO* x_out;
    T* b_coarse; // down leg
    const double* r64; // DOT: <r64, x_out> into *dot_out
    double* dot_partials;
    unsigned* dot_ticket;
    double* dot_out;
};

template <class T, class TC, bool UP, bool DOT, class TB = T, class TO = T>
__global__ void __launch_bounds__(BK_NT, 1) brick_leg_kernel(const BrickLegArgs<T, TC, TB, TO> a) {
    static_assert(UP || !DOT, "the dot product belongs to the last post-sweep");
    using G = BrickGeom<T>;
    constexpr int KP = G::KP, RZ = G::RZ, BZ = G::BZ, P = G::P, PZ = BK_R * P, R = BK_R, H = BK_H, B = BK_B;
    __shared__ __align__(16) T xs[RZ * PZ];
    __shared__ T ds[UP ? 1 : B * B * BZ], rs[UP ? 1 : B * B * BZ]; // own cells: D, then the residual
    const LevelOp<TC>& L = a.L;
    const int nx = L.nx, ny = L.ny, nz = L.nz;
    const size_t nxy = (size_t)nx * ny;
    const int t = threadIdx.x, m = t & 7, j = (t >> 3) & 15, kb = (t >> 7) * KP;
    const int x0 = blockIdx.x * B, y0 = blockIdx.y * B, z0 = blockIdx.z * BZ;
    const T dx2 = (T)L.dx2;
    // the pair's place in the grid (pairs start on even cells, and a periodic axis has an even count)
    const int wi = wrap_or_out(x0 - H + 2 * m, nx, L.per_x), wj = wrap_or_out(y0 - H + j, ny, L.per_y);
    const bool inxy = wi >= 0 && wj >= 0;
    // whether region cell (ai, j, k) is within r cells of the brick
    auto within = [&](int ai, int k, int r) {
        return ai >= H - r && ai < H + B + r && j >= H - r && j < H + B + r && k >= H - r && k < H + BZ + r;
    };
    // weights by colour (0: red): -x, +x, -y, +y, -z, +z, b dx^2 / D
    T w[2][KP][7], xv[2][KP];
    bool in[KP];
    int wk[KP];
#pragma unroll
    for (int q = 0; q < KP; ++q) {
        const int k = kb + q;
        wk[q] = wrap_or_out(z0 - H + k, nz, L.per_z);
        in[q] = inxy && wk[q] >= 0;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int o = (j + k + c) & 1; // the region's origin is even in j and k
#pragma unroll
            for (int f = 0; f < 7; ++f) w[c][q][f] = (T)0;
            xv[c][q] = (T)0;
            // the first half-sweep that updates the cell: reach 4 (red) or 3 (black) down, one less up
            if (in[q] && within(2 * m + o, k, (UP ? 3 : 4) - c)) {
                const size_t ci = (size_t)(wi + o) + (size_t)nx * wj + nxy * wk[q];
                T cxm, cxp, cym, cyp, czm, czp;
                cell_coefs<T>(L, wi + o, wj, wk[q], ci, cxm, cxp, cym, cyp, czm, czp);
                T D = cxm + cxp + cym + cyp + czm + czp;
                if (L.pin && ci == 0) D *= (T)2;
                const T inv = (T)1 / D;
                w[c][q][0] = cxm * inv;
                w[c][q][1] = cxp * inv;
                w[c][q][2] = cym * inv;
                w[c][q][3] = cyp * inv;
                w[c][q][4] = czm * inv;
                w[c][q][5] = czp * inv;
                w[c][q][6] = (T)a.b[ci] * dx2 * inv;
                if constexpr (!UP) {
                    if (within(2 * m + o, k, 0)) ds[(2 * m + o - H) + B * ((j - H) + B * (k - H))] = D;
                }
            }
            if constexpr (UP) {
                if (c == 1) { // red values are overwritten before they are read
                    T v = (T)0;
                    if (in[q]) {
                        const size_t ci = (size_t)(wi + o) + (size_t)nx * wj + nxy * wk[q];
                        v = a.x_in[ci] + __ldg(a.e_c + (size_t)(wi >> 1) + (size_t)a.ncx * ((size_t)(wj >> 1) + (size_t)a.ncy * (wk[q] >> 1)));
                    }
                    xs[k * PZ + j * P + 2 * m + o] = v;
                }
            } else {
                if (c == 0) { // the first red half-sweep, from x = 0
                    xv[0][q] = -w[0][q][6];
                    xs[k * PZ + j * P + 2 * m + o] = xv[0][q];
                }
            }
        }
    }
    __syncthreads();
    auto gs = [&](const T (&wt)[7], int f) -> T {
        return wt[0] * xs[f - 1] + wt[1] * xs[f + 1] + wt[2] * xs[f - P] + wt[3] * xs[f + P] + wt[4] * xs[f - PZ] +
               wt[5] * xs[f + PZ] - wt[6];
    };
    // one colour of a sweep on the cells within r of the brick
    auto half = [&](auto cc, int r) {
        constexpr int c = decltype(cc)::value;
#pragma unroll
        for (int q = 0; q < KP; ++q) {
            const int k = kb + q, ai = 2 * m + ((j + k + c) & 1);
            if (within(ai, k, r)) {
                const int f = k * PZ + j * P + ai;
                xv[c][q] = gs(w[c][q], f); // (zero weights outside a non-periodic axis: the ghost value)
                xs[f] = xv[c][q];
            }
        }
        __syncthreads();
    };
    using Red = std::integral_constant<int, 0>;
    using Black = std::integral_constant<int, 1>;
    if constexpr (UP) {
        half(Red{}, 3);
        half(Black{}, 2);
        half(Red{}, 1);
        half(Black{}, 0);
    } else {
        half(Black{}, 3);
        half(Red{}, 2);
        half(Black{}, 1);
        // residual of the brick's cells: r = D / dx^2 (x - x_GS)
        const T inv_dx2 = (T)L.inv_dx2;
#pragma unroll
        for (int q = 0; q < KP; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int k = kb + q, ai = 2 * m + ((j + k + c) & 1);
                if (within(ai, k, 0)) {
                    const int s = (ai - H) + B * ((j - H) + B * (k - H));
                    rs[s] = in[q] ? ds[s] * inv_dx2 * (xv[c][q] - gs(w[c][q], k * PZ + j * P + ai)) : (T)0;
                }
            }
        __syncthreads();
        const int nc = (B / 2) * (B / 2) * (BZ / 2);
        if (t < nc) {
            const int I = t % (B / 2), J = (t / (B / 2)) % (B / 2), K = t / ((B / 2) * (B / 2));
            const int gI = x0 / 2 + I, gJ = y0 / 2 + J, gK = z0 / 2 + K;
            if (gI < nx / 2 && gJ < ny / 2 && gK < nz / 2) {
                T acc = (T)0;
                // children in the order (000,100,010,110,001,101,011,111), restrict_3d.cu:38-49
#pragma unroll
                for (int d = 0; d < 8; ++d)
                    acc += rs[(2 * I + (d & 1)) + B * ((2 * J + ((d >> 1) & 1)) + B * (2 * K + (d >> 2)))];
                a.b_coarse[(size_t)gI + (size_t)(nx / 2) * ((size_t)gJ + (size_t)(ny / 2) * gK)] = acc / (T)8;
            }
        }
    }
    double dot = 0.0;
    if (m >= H / 2 && m < (H + B) / 2 && j >= H && j < H + B && inxy) {
#pragma unroll
        for (int q = 0; q < KP; ++q) {
            const int k = kb + q;
            // own planes inside the grid (a periodic copy past the top belongs to the brick that owns it)
            if (k < H || k >= H + BZ || z0 - H + k >= nz || x0 - H + 2 * m >= nx || y0 - H + j >= ny) continue;
            const int o = (j + k) & 1;
            const T va = o ? xv[1][q] : xv[0][q], vb = o ? xv[0][q] : xv[1][q];
            const size_t ci = (size_t)wi + (size_t)nx * wj + nxy * wk[q];
            a.x_out[ci] = (TO)va; // (scalar: a caller's z may start anywhere)
            a.x_out[ci + 1] = (TO)vb;
            if constexpr (DOT) dot += a.r64[ci] * (double)va + a.r64[ci + 1] * (double)vb;
        }
    }
    if constexpr (DOT) {
        double v[1] = {dot}, out[1];
        if (grid_sums<BK_NT, 1>(v, a.dot_partials, a.dot_ticket, gridDim.x * gridDim.y * gridDim.z, out)) *a.dot_out = out[0];
    }
}

} // namespace mf3d
