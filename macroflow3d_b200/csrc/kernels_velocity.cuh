// kernels_velocity.cuh -- Darcy face velocities from head, and the discrete mass balance.
//
// One kernel writes all three components (the reference launches 3 interior + 6 boundary
// kernels on the legacy default stream, src/physics/flow/velocity_from_head.cu:601-777).
// Each cell writes its three min-side faces; the plus faces are evaluated only at the max
// boundary, or for the mass balance, so an interior face is computed once.
// Formulas are the reference's: interior q = -[2 K_L K_R / (K_L + K_R)] (h_R - h_L)/dx;
// Dirichlet faces -K_c (h_c - h_bc)/(dx/2) (min side) and -K_c (h_bc - h_c)/(dx/2) (max side);
// Neumann 0; periodic faces use the wrapped neighbour (velocity_from_head.cu:102-381).
#pragma once
#include "kernels_setup.cuh"
#include "mf3d_device.cuh"

namespace mf3d {

// Flux through an interior (or periodic) face from cell L to cell R: -[2 K_L K_R / (K_L + K_R)]
// (h_R - h_L) / d, evaluated with one division (the reference's two differ in rounding only).
__device__ __forceinline__ double flux_lr(double KL, double KR, double HL, double HR, double d) {
    return (2.0 * KL * KR * (HL - HR)) / ((KL + KR) * d);
}

struct VelOut {
    double* U;
    double* V;
    double* W;
    int layout; // 0 compact MAC, 1 padded (nx+1)(ny+1)(nz+1)
};

__device__ __forceinline__ size_t u_idx(int layout, int i, int j, int k, int nx, int ny) {
    return layout ? (size_t)k * (ny + 1) * (nx + 1) + (size_t)j * (nx + 1) + i
                  : (size_t)i + (size_t)j * (nx + 1) + (size_t)k * (nx + 1) * ny;
}
__device__ __forceinline__ size_t v_idx(int layout, int i, int j, int k, int nx, int ny) {
    return layout ? (size_t)k * (ny + 1) * (nx + 1) + (size_t)j * (nx + 1) + i
                  : (size_t)i + (size_t)j * nx + (size_t)k * nx * (ny + 1);
}
__device__ __forceinline__ size_t w_idx(int layout, int i, int j, int k, int nx, int ny) {
    return layout ? (size_t)k * (ny + 1) * (nx + 1) + (size_t)j * (nx + 1) + i
                  : (size_t)i + (size_t)j * nx + (size_t)k * nx * ny;
}

// Flux through a boundary face of cell c on the min / max side of an axis; cw the wrapped
// neighbour for periodic.
__device__ __forceinline__ double face_min_bnd(const double* H, const double* K, size_t c, size_t cw, int type,
                                               double hbc, double d) {
    if (type == BC_DIRICHLET) return -K[c] * (H[c] - hbc) / (d * 0.5);
    if (type == BC_PERIODIC) return flux_lr(K[cw], K[c], H[cw], H[c], d);
    return 0.0;
}
__device__ __forceinline__ double face_max_bnd(const double* H, const double* K, size_t c, size_t cw, int type,
                                               double hbc, double d) {
    if (type == BC_DIRICHLET) return -K[c] * (hbc - H[c]) / (d * 0.5);
    if (type == BC_PERIODIC) return flux_lr(K[c], K[cw], H[c], H[cw], d);
    return 0.0;
}

constexpr int VEL_NT = 256;

// Writes U,V,W.  With MB also accumulates the mass balance:
// mb[0] = max_c |sum_f q_f A_f| (as ordered bits), mb[1] = Q_in (x=0), mb[2] = Q_out (x=L).
// A thread marches a column in z: K and h of the plane below stay in registers, those of the next
// plane are loaded before this plane's three divisions, the x neighbour comes from the lane beside, and
// every array has one running offset.  Per-cell index arithmetic and the branches of the
// boundary faces had bound it: 256^3 0.303 -> 0.175 ms (40 bytes a cell; 0.104 ms at the copy bandwidth).
template <bool MB>
__global__ void __launch_bounds__(VEL_NT, MB ? 2 : 3) velocity_kernel(int nx, int ny, int nz, double dx,
                                                          const double* __restrict__ H, const double* __restrict__ K,
                                                          BcDev bc, VelOut o, unsigned long long* mb_max,
                                                          double* partials, unsigned* ticket, double* mb_sums,
                                                          int zchunk) {
    const size_t nxy = (size_t)nx * ny;
    double qin = 0.0, qout = 0.0, mx = 0.0;
    const double A = dx * dx;
    const Col3 q = col3(nx, ny, nz, zchunk);
    const int i = q.i, j = q.j, lane = threadIdx.x;
    // lanes past the row stay in the loop (the shuffles need the whole warp) at a cell of the grid
    const bool own = q.ok;
    const int ic = min(i, nx - 1), jc = min(j, ny - 1);
    size_t c = (size_t)ic + (size_t)nx * jc + nxy * q.k0;
    size_t cu = u_idx(o.layout, ic, jc, q.k0, nx, ny), cv = v_idx(o.layout, ic, jc, q.k0, nx, ny);
    size_t cw = w_idx(o.layout, ic, jc, q.k0, nx, ny);
    const size_t su = u_idx(o.layout, 0, 0, 1, nx, ny), sv = v_idx(o.layout, 0, 0, 1, nx, ny);
    const size_t sw = w_idx(o.layout, 0, 0, 1, nx, ny), svy = v_idx(o.layout, 0, 1, 0, nx, ny);
    const bool x0 = ic == 0, x1 = ic == nx - 1, y0 = jc == 0, y1 = jc == ny - 1;
    const bool ldx = lane == 0 && !x0; // the lane that loads its x neighbour itself
    double Kb = 0.0, Hb = 0.0, Kn = 0.0, Hn = 0.0, Kwn = 0.0, Hwn = 0.0, Ksn = 0.0, Hsn = 0.0;
    auto fetch = [&](size_t cc) {
        Kn = __ldg(K + cc);
        Hn = __ldg(H + cc);
        if (ldx) Kwn = __ldg(K + cc - 1), Hwn = __ldg(H + cc - 1);
        if (!y0) Ksn = __ldg(K + cc - nx), Hsn = __ldg(H + cc - nx);
    };
    if (q.k0 < q.k1) {
        if (q.k0 > 0) Kb = __ldg(K + c - nxy), Hb = __ldg(H + c - nxy);
        fetch(c);
    }
    for (int k = q.k0; k < q.k1; ++k, c += nxy, cu += su, cv += sv, cw += sw) {
        const double Kc = Kn, Hc = Hn, Ks = Ksn, Hs = Hsn;
        double Kw = __shfl_up_sync(0xffffffffu, Kc, 1), Hw = __shfl_up_sync(0xffffffffu, Hc, 1);
        if (ldx) Kw = Kwn, Hw = Hwn;
        if (k + 1 < q.k1) fetch(c + nxy);
        const double u0 = x0 ? face_min_bnd(H, K, c, c + (nx - 1), bc.type[0], bc.value[0], dx)
                             : flux_lr(Kw, Kc, Hw, Hc, dx);
        const double v0 = y0 ? face_min_bnd(H, K, c, c + (size_t)(ny - 1) * nx, bc.type[2], bc.value[2], dx)
                             : flux_lr(Ks, Kc, Hs, Hc, dx);
        const double w0 = k == 0 ? face_min_bnd(H, K, c, c + (size_t)(nz - 1) * nxy, bc.type[4], bc.value[4], dx)
                                 : flux_lr(Kb, Kc, Hb, Hc, dx);
        Kb = Kc;
        Hb = Hc;
        if (own) {
            o.U[cu] = u0;
            o.V[cv] = v0;
            o.W[cw] = w0;
            // plus faces: at the max boundary (written here), and for the mass balance the
            // neighbour's min face, with the same arithmetic as that neighbour's store
            double u1 = 0.0, v1 = 0.0, w1 = 0.0;
            if (x1) {
                u1 = face_max_bnd(H, K, c, c - (nx - 1), bc.type[1], bc.value[1], dx);
                o.U[cu + 1] = u1;
            } else if (MB) {
                u1 = flux_lr(Kc, K[c + 1], Hc, H[c + 1], dx);
            }
            if (y1) {
                v1 = face_max_bnd(H, K, c, c - (size_t)(ny - 1) * nx, bc.type[3], bc.value[3], dx);
                o.V[cv + svy] = v1;
            } else if (MB) {
                v1 = flux_lr(Kc, K[c + nx], Hc, H[c + nx], dx);
            }
            if (k == nz - 1) {
                w1 = face_max_bnd(H, K, c, c - (size_t)(nz - 1) * nxy, bc.type[5], bc.value[5], dx);
                o.W[cw + sw] = w1;
            } else if (MB) {
                w1 = flux_lr(Kc, K[c + nxy], Hc, H[c + nxy], dx);
            }
            if (MB) {
                const double d = ((u1 - u0) + (v1 - v0) + (w1 - w0)) * A;
                mx = fmax(mx, fabs(d));
                if (x0) qin += u0 * A;
                if (x1) qout += u1 * A;
            }
        }
    }
    if (MB) {
        double v[2] = {qin, qout}, out[2];
        // max: non-negative doubles order like their bit patterns
        for (int ofs = 16; ofs > 0; ofs >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, ofs));
        if (threadIdx.x == 0) atomicMax(mb_max, (unsigned long long)__double_as_longlong(mx)); // lane 0 of each warp row
        if (grid_sums<VEL_NT, 2>(v, partials, ticket, gridDim.x * gridDim.y * gridDim.z, out)) {
            mb_sums[0] = out[0];
            mb_sums[1] = out[1];
        }
    }
}

// ---------------------------------------------------------------------------------------
// Velocity diagnostics at cell centres (compute_velocity_diagnostics,
// src/physics/flow/velocity_diagnostics.cu:48-179): the divergence of every cell, and at the
// interior cells (1 <= i <= nx-2, likewise j, k; none when a dimension is below 3) the curl of
// the face-averaged cell velocity by centred differences, its magnitude and the helicity
// u . curl u; zero elsewhere.  Any output may be null.  With stats != null the kernel also
// reduces min / max / sum of the three fields (deterministic: per-block partials combined in
// block order by the last block); stats[9] = min, max, mean of div, |omega|, helicity.
// A CTA marches a 32 x 8 column tile in z.  Each thread forms the cell velocity of its column once per plane
// (five loads, one plane ahead) and keeps the planes below and above in registers; the x and y neighbours
// come from shared memory, where 80 threads also put the cells beside the tile.  Thirty loads per cell
// with their index arithmetic had bound it: 201 x 150 x 99, padded: 0.145 -> 0.068 ms.
// ---------------------------------------------------------------------------------------
constexpr int VD_NT = 256;

__device__ __forceinline__ void vd_block_reduce(double (&mn)[3], double (&mx)[3], double (&sm)[3], double* red) {
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    for (int o = 16; o > 0; o >>= 1)
        for (int q = 0; q < 3; ++q) {
            mn[q] = fmin(mn[q], __shfl_down_sync(0xffffffffu, mn[q], o));
            mx[q] = fmax(mx[q], __shfl_down_sync(0xffffffffu, mx[q], o));
            sm[q] += __shfl_down_sync(0xffffffffu, sm[q], o);
        }
    const int w = tid >> 5, l = tid & 31;
    if (l == 0)
        for (int q = 0; q < 3; ++q) {
            red[(3 * q) * (VD_NT / 32) + w] = mn[q];
            red[(3 * q + 1) * (VD_NT / 32) + w] = mx[q];
            red[(3 * q + 2) * (VD_NT / 32) + w] = sm[q];
        }
    __syncthreads();
    if (tid == 0)
        for (int q = 0; q < 3; ++q) {
            double a = red[(3 * q) * (VD_NT / 32)], b = red[(3 * q + 1) * (VD_NT / 32)], c = 0.0;
            for (int i = 0; i < VD_NT / 32; ++i) {
                a = fmin(a, red[(3 * q) * (VD_NT / 32) + i]);
                b = fmax(b, red[(3 * q + 1) * (VD_NT / 32) + i]);
                c += red[(3 * q + 2) * (VD_NT / 32) + i];
            }
            mn[q] = a, mx[q] = b, sm[q] = c;
        }
    __syncthreads();
}

__global__ void __launch_bounds__(VD_NT, 3) velocity_diag_kernel(int nx, int ny, int nz, double inv_dx, int layout,
                                                              const double* __restrict__ U,
                                                              const double* __restrict__ V,
                                                              const double* __restrict__ W, double* div,
                                                              double* omag, double* hel, double* partials,
                                                              unsigned* ticket, double* stats, int zchunk) {
    __shared__ double red[9 * (VD_NT / 32)];
    __shared__ bool s_last;
    constexpr int TX = 32, TY = VD_NT / 32, PW = TX + 2;
    __shared__ double su[2][TY + 2][PW], sv[2][TY + 2][PW], sw[2][TY + 2][PW]; // cell velocities of a plane
    const size_t nxy = (size_t)nx * ny;
    const double inv2 = 0.5 * inv_dx;
    const bool curl = nx >= 3 && ny >= 3 && nz >= 3;
    double mn[3], mx[3], sm[3];
    for (int q = 0; q < 3; ++q) mn[q] = INFINITY, mx[q] = -INFINITY, sm[q] = 0.0;
    const Col3 q = col3(nx, ny, nz, zchunk);
    const int i = q.i, j = q.j, tx = threadIdx.x, ty = threadIdx.y;
    const size_t suy = u_idx(layout, 0, 1, 0, nx, ny), suz = u_idx(layout, 0, 0, 1, nx, ny);
    const size_t svy = v_idx(layout, 0, 1, 0, nx, ny), svz = v_idx(layout, 0, 0, 1, nx, ny);
    const size_t swy = w_idx(layout, 0, 1, 0, nx, ny), swz = w_idx(layout, 0, 0, 1, nx, ny);
    // a second cell beside the tile: threads 0-31 the row below, 32-63 the row above (u and w are read
    // there), 64-71 the column left, 72-79 right (v and w)
    int ei = 0, ej = 0, el = 0;
    const int t = tx + TX * ty;
    if (t < 2 * TX) ei = i - tx + (t & 31), ej = j - ty + (t < TX ? -1 : TY), el = 1;
    else if (t < 2 * TX + 2 * TY) ei = i - tx + (t < 2 * TX + TY ? -1 : TX), ej = j - ty + (t & 7), el = 2;
    const bool eok = el != 0 && curl && ei >= 0 && ei < nx && ej >= 0 && ej < ny;
    const int ey = ej - (j - ty) + 1, ex = ei - (i - tx) + 1; // its place in the plane
    const size_t ou = q.ok ? (size_t)i + suy * j : 0, ov = q.ok ? (size_t)i + svy * j : 0, ow = q.ok ? (size_t)i + swy * j : 0;
    // u (el 1) or v (el 2) of the second cell as a pair of faces da apart, and w
    const double* eb = el == 1 ? U : V;
    const size_t ea = eok ? (el == 1 ? (size_t)ei + suy * ej : (size_t)ei + svy * ej) : 0, eaz = el == 1 ? suz : svz;
    const size_t eda = el == 1 ? 1 : svy, ew = eok ? (size_t)ei + swy * ej : 0;
    // faces of the next plane; w faces: the next plane's upper one
    double nU = 0, nUp = 0, nV = 0, nVp = 0, nW = 0, eA = 0, eAp = 0, eW = 0;
    auto fetch = [&](int k) {
        if (q.ok) {
            nU = __ldg(U + ou + suz * k), nUp = __ldg(U + ou + suz * k + 1);
            nV = __ldg(V + ov + svz * k), nVp = __ldg(V + ov + svz * k + svy);
            nW = __ldg(W + ow + swz * (k + 1));
        }
        if (eok) {
            eA = __ldg(eb + ea + eaz * k), eAp = __ldg(eb + ea + eaz * k + eda);
            eW = __ldg(W + ew + swz * (k + 1));
        }
    };
    double um = 0, vm = 0, Wk = 0, eWk = 0; // cell velocities of the plane below, lower w faces
    if (q.k0 < q.k1) {
        if (q.k0 > 0 && q.ok) {
            const size_t k = q.k0 - 1;
            um = 0.5 * (__ldg(U + ou + suz * k) + __ldg(U + ou + suz * k + 1));
            vm = 0.5 * (__ldg(V + ov + svz * k) + __ldg(V + ov + svz * k + svy));
        }
        if (q.ok) Wk = __ldg(W + ow + swz * q.k0);
        if (eok) eWk = __ldg(W + ew + swz * q.k0);
        fetch(q.k0);
    }
    for (int k = q.k0; k < q.k1; ++k) {
        const int bf = k & 1;
        const double Ui = nU, Uip = nUp, Vj = nV, Vjp = nVp, Wkp = nW;
        const double u0 = 0.5 * (Ui + Uip), v0 = 0.5 * (Vj + Vjp), w0 = 0.5 * (Wk + Wkp);
        su[bf][ty + 1][tx + 1] = u0;
        sv[bf][ty + 1][tx + 1] = v0;
        sw[bf][ty + 1][tx + 1] = w0;
        if (eok) {
            (el == 1 ? su : sv)[bf][ey][ex] = 0.5 * (eA + eAp);
            sw[bf][ey][ex] = 0.5 * (eWk + eW);
            eWk = eW;
        }
        if (k + 1 < nz) fetch(k + 1);
        __syncthreads(); // (the other buffer's plane was read before the last barrier)
        if (q.ok) {
            const size_t c = (size_t)i + (size_t)nx * j + nxy * k;
            const double d = (Uip - Ui) * inv_dx + (Vjp - Vj) * inv_dx + (Wkp - Wk) * inv_dx;
            double om = 0.0, he = 0.0;
            if (curl && i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2 && k >= 1 && k <= nz - 2) {
                const double dwdy = (sw[bf][ty + 2][tx + 1] - sw[bf][ty][tx + 1]) * inv2;
                const double dvdz = (0.5 * (nV + nVp) - vm) * inv2;
                const double dudz = (0.5 * (nU + nUp) - um) * inv2;
                const double dwdx = (sw[bf][ty + 1][tx + 2] - sw[bf][ty + 1][tx]) * inv2;
                const double dvdx = (sv[bf][ty + 1][tx + 2] - sv[bf][ty + 1][tx]) * inv2;
                const double dudy = (su[bf][ty + 2][tx + 1] - su[bf][ty][tx + 1]) * inv2;
                const double ox = dwdy - dvdz, oy = dudz - dwdx, oz = dvdx - dudy;
                om = sqrt(ox * ox + oy * oy + oz * oz);
                he = u0 * ox + v0 * oy + w0 * oz;
            }
            if (div) div[c] = d;
            if (omag) omag[c] = om;
            if (hel) hel[c] = he;
            const double f[3] = {d, om, he};
            for (int r = 0; r < 3; ++r) mn[r] = fmin(mn[r], f[r]), mx[r] = fmax(mx[r], f[r]), sm[r] += f[r];
        }
        um = u0, vm = v0, Wk = Wkp;
    }
    if (!stats) return;
    const int nb = gridDim.x * gridDim.y * gridDim.z;
    const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    vd_block_reduce(mn, mx, sm, red);
    if (tid == 0) {
        for (int r = 0; r < 3; ++r) {
            partials[(size_t)(3 * r) * nb + bid] = mn[r];
            partials[(size_t)(3 * r + 1) * nb + bid] = mx[r];
            partials[(size_t)(3 * r + 2) * nb + bid] = sm[r];
        }
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == (unsigned)nb - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int r = 0; r < 3; ++r) mn[r] = INFINITY, mx[r] = -INFINITY, sm[r] = 0.0;
    // the last block: partials in block order, each thread a strided subset, then the block
    for (int b = tid; b < nb; b += VD_NT)
        for (int r = 0; r < 3; ++r) {
            mn[r] = fmin(mn[r], __ldcg(partials + (size_t)(3 * r) * nb + b));
            mx[r] = fmax(mx[r], __ldcg(partials + (size_t)(3 * r + 1) * nb + b));
            sm[r] += __ldcg(partials + (size_t)(3 * r + 2) * nb + b);
        }
    vd_block_reduce(mn, mx, sm, red);
    if (tid == 0) {
        const double n = (double)nxy * nz;
        for (int r = 0; r < 3; ++r) {
            stats[3 * r] = mn[r];
            stats[3 * r + 1] = mx[r];
            stats[3 * r + 2] = sm[r] / n;
        }
        *ticket = 0u;
    }
}

} // namespace mf3d
