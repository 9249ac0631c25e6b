// kernels_kfield.cuh -- log-normal K by the randomization (spectral) method.
//
// lnK(x) = sigma / sqrt(N) * sum_m (a_m sin(k_m . x) + b_m cos(k_m . x)) at cell centres,
// K = exp(lnK + ln K_g) (src/physics/stochastic/stochastic.cu:180-260).  The phase is a sum of one term
// per axis, so with p = k_x x_i and q = k_y y_j + k_z z_k
//   a sin(p + q) + b cos(p + q) = sin p (a cos q - b sin q) + cos p (a sin q + b cos q):
// the field is a matrix product, (rows (j, k)) x (2 N) times (2 N) x (columns i).  kfield_tables_kernel
// evaluates the sines and cosines once per mode and coordinate; kfield_kernel forms the rows' factors
// from the tables of y and z (four multiply-adds per mode and row) in shared memory and multiplies on
// the FP64 tensor cores (m8n8k4, FP64 accumulation).
// Bound by FP64: 2 multiply-adds per mode and cell, 0.23 ms for 128^3 cells and 1000 modes at 64 per SM and
// cycle.  Measured there: 0.365 ms (1.35 ms when every
// thread advanced a run of 16 cells by rotations, six operations per mode and cell; the error against 64-bit
// sums fell from 1.3e-13 to 6e-15).  16 modes staged at a time, with three CTAs on an SM: 0.474 ms.
#pragma once
#include "mf3d_device.cuh"

namespace mf3d {

constexpr int KF_MC = 8;            // modes staged at a time (16 rows of the inner dimension): four CTAs on an SM
constexpr int KF_NT = 128;          // 4 warps
constexpr int KF_COLS = 32;         // columns per warp
constexpr int KF_K = 2 * KF_MC;
// row pitch of the staged operands in doubles: 4 mod 16, so that the 16 lanes of a half-warp's fragment
// load (4 inner x 4 outer) hit different banks
__host__ __device__ constexpr int kf_pitch(int n) { return n + 4; }
template <int MT, int RW, int CW> struct KfGeom {
    static_assert(RW * CW * 32 == KF_NT, "four warps");
    static constexpr int ROWS = 8 * MT * RW, COLS = KF_COLS * CW;
    static constexpr int PA = kf_pitch(ROWS), PB = kf_pitch(COLS);
    static constexpr size_t STAGE = (size_t)KF_K * (PA + PB);
    static constexpr size_t SMEM = 2 * STAGE * sizeof(double);
};

// The part of a field one launch evaluates: cells [ox, ox + nx) x [oy, oy + ny) x [oz, oz + nz) of a field
// of row length NX and NY rows a plane, and the modes [m0, m0 + n) of all; the sums of the modes before
// m0 are in `out` already (m0 > 0), and the last part applies the scale and the exponential.
struct KfPart {
    int ox, oy, oz, nx, ny, nz, NX, NY;
    int m0, n, last;
};

// Tables of a part: tx[2 m + {0, 1}][nxp] = sin, cos of k_x x_i (zero past nx), ty[m][ny] = sin, cos pairs
// of k_y y_j, uv[m][nz] = (a cos - b sin, a sin + b cos) of k_z z_k; zeros for the modes n .. mp.
__global__ void kfield_tables_kernel(const KfPart w, double dx, int n_modes, int mp, int nxp,
                                     const double* __restrict__ modes0, double* __restrict__ tx,
                                     double2* __restrict__ ty, double2* __restrict__ uv) {
    const int nx = w.nx, ny = w.ny, nz = w.nz, len = nxp + ny + nz;
    const double* modes = modes0 + w.m0;
    const size_t n = (size_t)mp * len;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int m = (int)(e / len), c = (int)(e % len);
        const bool live = m < w.n;
        double s = 0.0, co = 0.0;
        if (c < nxp) {
            if (live && c < nx) sincos(modes[m] * (dx * ((w.ox + c) + 0.5)), &s, &co);
            tx[(size_t)(2 * m) * nxp + c] = s;
            tx[(size_t)(2 * m + 1) * nxp + c] = co;
        } else if (c < nxp + ny) {
            const int j = c - nxp;
            if (live) sincos(modes[n_modes + m] * (dx * ((w.oy + j) + 0.5)), &s, &co);
            ty[(size_t)m * ny + j] = make_double2(s, co);
        } else {
            const int k = c - nxp - ny;
            double u = 0.0, v = 0.0;
            if (live) {
                const double a = modes[3 * (size_t)n_modes + m], b = modes[4 * (size_t)n_modes + m];
                sincos(modes[2 * (size_t)n_modes + m] * (dx * ((w.oz + k) + 0.5)), &s, &co);
                u = a * co - b * s;
                v = a * s + b * co;
            }
            uv[(size_t)m * nz + k] = make_double2(u, v);
        }
    }
}

__device__ __forceinline__ void kf_mma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// MT x 8 rows by 32 columns per warp, RW x CW warps; rows are (j, k) pairs, j fastest.
template <int MT, int RW, int CW>
__global__ void __launch_bounds__(KF_NT) kfield_kernel(const KfPart w, int mp, int nxp, const double* __restrict__ tx,
                                                       const double2* __restrict__ ty, const double2* __restrict__ uv,
                                                       double scale, double log_kg, int want_exp,
                                                       double* __restrict__ out) {
    const int nx = w.nx, ny = w.ny, nz = w.nz;
    using G = KfGeom<MT, RW, CW>;
    extern __shared__ __align__(16) double kf_sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const size_t nrows = (size_t)ny * nz, row0 = (size_t)blockIdx.x * G::ROWS;
    const int col0 = blockIdx.y * G::COLS;
    // the row this thread stages, of every (NT / ROWS)-th mode
    constexpr int RT = G::ROWS < KF_NT ? G::ROWS : KF_NT, MS = KF_NT / RT;
    const size_t sr = row0 + (tid % RT);
    const bool sin_ = sr < nrows;
    const int sj = sin_ ? (int)(sr % ny) : 0, sk = sin_ ? (int)(sr / ny) : 0;
    auto stage_b = [&](int m0, int buf) {
        double* B = kf_sm + buf * G::STAGE + (size_t)KF_K * G::PA;
        for (int q = tid; q < KF_K * (G::COLS / 2); q += KF_NT) {
            const int kk = q / (G::COLS / 2), c = 2 * (q % (G::COLS / 2));
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(B + kk * G::PB + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                         "l"(tx + (size_t)(2 * m0 + kk) * nxp + col0 + c)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto stage_a = [&](int m0, int buf) {
        double* A = kf_sm + buf * G::STAGE;
#pragma unroll 4
        for (int q = tid / RT; q < KF_MC; q += MS) {
            const double2 y = __ldg(ty + (size_t)(m0 + q) * ny + sj), z = __ldg(uv + (size_t)(m0 + q) * nz + sk);
            A[(2 * q) * G::PA + tid % RT] = z.x * y.y - z.y * y.x;
            A[(2 * q + 1) * G::PA + tid % RT] = z.y * y.y + z.x * y.x;
        }
    };
    const int wr = (warp / CW) * 8 * MT, wc = (warp % CW) * KF_COLS, g = lane >> 2, t = lane & 3;
    double acc[MT][4][2];
#pragma unroll
    for (int r = 0; r < MT; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;
    stage_b(0, 0);
    stage_a(0, 0);
    int buf = 0;
    for (int m0 = 0; m0 < mp; m0 += KF_MC, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads(); // this chunk is staged, the other buffer's products are done
        if (m0 + KF_MC < mp) {
            stage_b(m0 + KF_MC, buf ^ 1);
            stage_a(m0 + KF_MC, buf ^ 1);
        }
        const double* A = kf_sm + buf * G::STAGE;
        const double* B = A + (size_t)KF_K * G::PA;
#pragma unroll
        for (int k4 = 0; k4 < KF_K; k4 += 4) {
            double a[MT], b[4];
#pragma unroll
            for (int r = 0; r < MT; ++r) a[r] = A[(k4 + t) * G::PA + wr + 8 * r + g];
#pragma unroll
            for (int c = 0; c < 4; ++c) b[c] = B[(k4 + t) * G::PB + wc + 8 * c + g];
#pragma unroll
            for (int r = 0; r < MT; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) kf_mma(acc[r][c], a[r], b[c]);
        }
    }
#pragma unroll
    for (int r = 0; r < MT; ++r) {
        const size_t row = row0 + wr + 8 * r + g;
        if (row >= nrows) continue;
        const size_t o = (size_t)w.ox + (size_t)w.NX * ((size_t)(w.oy + (int)(row % ny)) + (size_t)w.NY * (w.oz + (int)(row / ny)));
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = col0 + wc + 8 * c + 2 * t + h;
                if (i < nx) {
                    double v = acc[r][c][h];
                    if (w.m0 > 0) v += out[o + i];
                    if (w.last) {
                        v *= scale;
                        if (want_exp) v = exp(v + log_kg);
                    }
                    out[o + i] = v;
                }
            }
    }
}

// The same part without tables, a cell per thread: where the device has no room for them (a sine and a cosine per
// mode and cell).
__global__ void __launch_bounds__(256) kfield_direct_kernel(const KfPart w, double dx, int n_modes,
                                                            const double* __restrict__ modes, double scale,
                                                            double log_kg, int want_exp, double* __restrict__ out) {
    const size_t n = (size_t)w.nx * w.ny * w.nz;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int i = w.ox + (int)(e % w.nx), j = w.oy + (int)((e / w.nx) % w.ny), k = w.oz + (int)(e / ((size_t)w.nx * w.ny));
        const double x = dx * (i + 0.5), y = dx * (j + 0.5), z = dx * (k + 0.5);
        double v = 0.0;
        for (int m = 0; m < n_modes; ++m) {
            const double* q = modes + m;
            double s, c;
            sincos(q[0] * x + q[(size_t)n_modes] * y + q[2 * (size_t)n_modes] * z, &s, &c);
            v += q[3 * (size_t)n_modes] * s + q[4 * (size_t)n_modes] * c;
        }
        v *= scale;
        if (want_exp) v = exp(v + log_kg);
        out[(size_t)i + (size_t)w.NX * ((size_t)j + (size_t)w.NY * k)] = v;
    }
}

} // namespace mf3d
