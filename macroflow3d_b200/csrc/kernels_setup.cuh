// kernels_setup.cuh -- per-K setup: face coefficients, K coarsening, right-hand side and
// initial guess.  Runs once per conductivity field.
#pragma once
#include <type_traits>

#include "mf3d_device.cuh"

namespace mf3d {

struct BcDev {
    int type[6];
    double value[6];
};

// Harmonic mean exactly as the reference evaluates it
// (src/multigrid/common/mg_conventions.cuh:133-135); symmetric in its arguments bit-for-bit.
__device__ __forceinline__ double hmean_ref(double a, double b) { return 2.0 / (1.0 / a + 1.0 / b); }

template <class TC> __device__ __forceinline__ TC store_coef(double v);
template <> __device__ __forceinline__ double store_coef<double>(double v) { return v; }
template <> __device__ __forceinline__ float store_coef<float>(double v) { return (float)v; }
template <> __device__ __forceinline__ __nv_bfloat16 store_coef<__nv_bfloat16>(double v) {
    return __float2bfloat16_rn((float)v);
}

template <class TC> struct FacePtrs {
    TC *cx, *cy, *cz, *bxm, *bym, *bzm; // null: not stored
};

// Face coefficients of one level from its cell K (FP64), in one or two precisions; the second set is
// scaled by `scale` (1 unless the level stores bf16 with a power-of-two scale).  The values are hmean_ref's to
// the last bit with five divisions a cell instead of nine for each precision: a thread marches in z and
// keeps its cell's 1 / K for the plane above, the x neighbour's comes from the lane beside.  256^3, FP64 and
// FP32: 0.40 ms in two launches -> 0.23 ms in one.
template <class TA, class TB>
__global__ void __launch_bounds__(256) faces_kernel(int nx, int ny, int nz, const double* __restrict__ K, BcDev bc,
                                                    double scale, const FacePtrs<TA> A, const FacePtrs<TB> B,
                                                    int zchunk) {
    const size_t nxy = (size_t)nx * ny;
    const Col3 q = col3(nx, ny, nz, zchunk);
    const int lane = threadIdx.x, i = min(q.i, nx - 1), j = min(q.j, ny - 1);
    const bool x1 = i == nx - 1, y1 = j == ny - 1, own = q.ok;
    size_t c = (size_t)i + (size_t)nx * j + nxy * q.k0;
    double Kc = 0.0, rc = 0.0;
    if (q.k0 < q.k1) Kc = __ldg(K + c), rc = 1.0 / Kc;
    auto bnd = [&](int type) { return type == BC_DIRICHLET ? 2.0 * Kc : 0.0; };
    for (int k = q.k0; k < q.k1; ++k, c += nxy) {
        const bool z1 = k == nz - 1;
        const double Kn = z1 ? 0.0 : __ldg(K + c + nxy), rn = z1 ? 0.0 : 1.0 / Kn;
        double rx = __shfl_down_sync(0xffffffffu, rc, 1);
        if (x1) {
            if (bc.type[1] == BC_PERIODIC) rx = 1.0 / __ldg(K + c - (nx - 1));
        } else if (lane == 31) {
            rx = 1.0 / __ldg(K + c + 1);
        }
        const bool px = !x1 || bc.type[1] == BC_PERIODIC, py = !y1 || bc.type[3] == BC_PERIODIC;
        const bool pz = !z1 || bc.type[5] == BC_PERIODIC;
        double ry = 0.0, rz = rn;
        if (py) ry = 1.0 / __ldg(K + (y1 ? c - (size_t)(ny - 1) * nx : c + nx));
        if (z1 && pz) rz = 1.0 / __ldg(K + c - (size_t)(nz - 1) * nxy);
        const double vx = px ? 2.0 / (rc + rx) : bnd(bc.type[1]), vy = py ? 2.0 / (rc + ry) : bnd(bc.type[3]);
        const double vz = pz ? 2.0 / (rc + rz) : bnd(bc.type[5]);
        if (own) {
            const size_t ix = (size_t)j + (size_t)ny * k, iy = (size_t)i + (size_t)nx * k, iz = (size_t)i + (size_t)nx * j;
            auto put = [&](const auto& P, double s) {
                using TC = typename std::remove_pointer<decltype(P.cx)>::type;
                P.cx[c] = store_coef<TC>(vx * s);
                P.cy[c] = store_coef<TC>(vy * s);
                P.cz[c] = store_coef<TC>(vz * s);
                // minus boundary faces
                if (i == 0) P.bxm[ix] = store_coef<TC>(bnd(bc.type[0]) * s);
                if (j == 0) P.bym[iy] = store_coef<TC>(bnd(bc.type[2]) * s);
                if (k == 0) P.bzm[iz] = store_coef<TC>(bnd(bc.type[4]) * s);
            };
            if (A.cx) put(A, 1.0);
            if (B.cx) put(B, scale);
        }
        Kc = Kn;
        rc = rn;
    }
}

// Geometric mean of the 8 children, src/physics/flow/coarsen_K.cu:15-53 (same order).
__global__ void coarsen_kernel(int NX, int NY, int NZ, const double* __restrict__ Kf, double* __restrict__ Kc,
                               int zchunk) {
    const int Nx = 2 * NX;
    const size_t stride = (size_t)Nx * 2 * NY;
    const Col3 q = col3(NX, NY, NZ, zchunk);
    if (!q.ok) return;
    const int I = q.i, J = q.j;
    for (int Kk = q.k0; Kk < q.k1; ++Kk) {
        const size_t C = (size_t)I + (size_t)NX * J + (size_t)NX * NY * Kk;
        const size_t i000 = (size_t)(2 * I) + (size_t)Nx * (2 * J) + stride * (2 * Kk);
        const size_t i001 = i000 + stride;
        const double ls = log(Kf[i000]) + log(Kf[i000 + 1]) + log(Kf[i000 + Nx]) + log(Kf[i000 + 1 + Nx]) +
                          log(Kf[i001]) + log(Kf[i001 + 1]) + log(Kf[i001 + Nx]) + log(Kf[i001 + 1 + Nx]);
        Kc[C] = exp(ls / 8.0);
    }
}

// b: Dirichlet contributions -2 h_bc K_c / dx^2 (src/physics/flow/rhs_head.cu:21-194, faces
// in the order xmin..zmax); K is read on those faces only.
__global__ void rhs_kernel(int nx, int ny, int nz, double dx, const double* __restrict__ K, BcDev bc,
                           double* __restrict__ b, int zchunk) {
    const double inv_dx2 = 1.0 / (dx * dx);
    const Col3 q = col3(nx, ny, nz, zchunk);
    if (!q.ok) return;
    const int i = q.i, j = q.j;
    const bool fx0 = i == 0 && bc.type[0] == BC_DIRICHLET, fx1 = i == nx - 1 && bc.type[1] == BC_DIRICHLET;
    const bool fy0 = j == 0 && bc.type[2] == BC_DIRICHLET, fy1 = j == ny - 1 && bc.type[3] == BC_DIRICHLET;
    size_t c = (size_t)i + (size_t)nx * j + (size_t)nx * ny * q.k0;
    for (int k = q.k0; k < q.k1; ++k, c += (size_t)nx * ny) {
        const bool fz0 = k == 0 && bc.type[4] == BC_DIRICHLET, fz1 = k == nz - 1 && bc.type[5] == BC_DIRICHLET;
        double v = 0.0;
        if (fx0 | fx1 | fy0 | fy1 | fz0 | fz1) {
            const double Kc = K[c];
            if (fx0) v -= 2.0 * bc.value[0] * Kc * inv_dx2;
            if (fx1) v -= 2.0 * bc.value[1] * Kc * inv_dx2;
            if (fy0) v -= 2.0 * bc.value[2] * Kc * inv_dx2;
            if (fy1) v -= 2.0 * bc.value[3] * Kc * inv_dx2;
            if (fz0) v -= 2.0 * bc.value[4] * Kc * inv_dx2;
            if (fz1) v -= 2.0 * bc.value[5] * Kc * inv_dx2;
        }
        b[c] = v;
    }
}

// The initial guess (src/physics/flow/solve_head.cu:29-73): linear in x when both x faces are Dirichlet,
// else 0.
struct Guess {
    double h0, dh; // value at x = 0 and difference over the domain
};
inline Guess make_guess(const BcDev& bc) {
    const bool lin = bc.type[0] == BC_DIRICHLET && bc.type[1] == BC_DIRICHLET;
    return lin ? Guess{bc.value[0], bc.value[1] - bc.value[0]} : Guess{0.0, 0.0};
}
__device__ __forceinline__ double guess_at(const Guess& g, int i, int nx) {
    return g.h0 + g.dh * (((double)i + 0.5) / (double)nx);
}
__global__ void guess_kernel(int nx, size_t nrows, const Guess g, double* __restrict__ h) {
    // a warp per row: one division a cell and no index division
    const int lane = threadIdx.x & 31;
    for (size_t row = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); row < nrows;
         row += (size_t)gridDim.x * (blockDim.x >> 5))
        for (int i = lane; i < nx; i += 32) h[row * nx + i] = guess_at(g, i, nx);
}

template <class TO, class TI>
__global__ void convert_kernel(size_t n, const TI* __restrict__ in, TO* __restrict__ out) {
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
        out[c] = (TO)in[c];
}

} // namespace mf3d
