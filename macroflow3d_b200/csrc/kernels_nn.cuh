// kernels_nn.cuh -- kernels of the learned warm start: a small 3-D convolutional
// encoder-decoder (BF16 activations and weights, FP32 accumulation) whose output is the PCG
// initial guess.  No counterpart in the reference, whose initial guess is the x-linear head
// (src/physics/flow/solve_head.cu:29-73).
//
// Layout: activations are voxel-major with channels innermost ("NDHWC"): element (v, c) at
// v * C + c, v = i + nx (j + ny k).  Weights of a 3x3x3 convolution are [cout][27][cin] with
// tap t = (dz+1)*9 + (dy+1)*3 + (dx+1).
//
// conv3d_brick_kernel: implicit GEMM on the 5th-generation tensor cores.  D[v][co] =
// sum_{t, ci} X[v + off(t)][ci] W[co][t][ci]: M = 128 voxels, N = output channels of three output planes,
// K = 27 cin in steps of 16 channels, FP32 accumulators in TMEM.  The data gradient of a convolution is
// the same kernel on the output gradient with the weights flipped in the taps and transposed in the
// channels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels_pcg.cuh"

namespace mf3d {
namespace nn {

constexpr int CONV_TM = 128;   // voxels per tile (UMMA M)
constexpr int CONV_MAXC = 128; // channel limit (multiples of 16)

// ---- tcgen05 helpers ------------------------------------------------------------------
__device__ __forceinline__ uint32_t sm_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// One lane of the warp, the same one for the same (full) mask.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r;
}
// D(tmem) (+)= A(smem desc) * B(smem desc)^T, kind::f16 (BF16 inputs, FP32 accumulate), called by a whole warp in
// uniform control flow and issued by its elected lane: the descriptors then stay in uniform registers.  From one lane's own branch every product
// moved its descriptors there first, which took longer than the product (16 -> 16 channels at 128^3:
// 127 cycles a product).  Descriptors as (low, high) words; only the low one carries the start address.
__device__ __forceinline__ void umma_bf16_warp(uint32_t d_tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                               uint32_t idesc, uint32_t accumulate, uint32_t leader) {
    asm volatile("{\n .reg .pred p, q;\n .reg .b64 da, db;\n setp.ne.b32 p, %6, 0;\n setp.ne.b32 q, %7, 0;\n"
                 " mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n"
                 " @q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}" ::"r"(d_tmem),
                 "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate), "r"(leader)
                 : "memory");
}
// arrive on an mbarrier once every tcgen05.mma this thread issued before has completed
__device__ __forceinline__ void umma_commit_warp(uint64_t* bar, uint32_t leader) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
                 " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(sm_u32(bar)),
                 "r"(leader)
                 : "memory");
}
// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 columns of this thread's TMEM lane = 0; complete after tmem_wait_st
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
                 "r"(0u)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void nn_mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sm_u32(bar)), "r"(count) : "memory");
}
// bounded wait on an mbarrier phase; false when it gave up.  Each try suspends the thread for
// up to 2 us unless the phase completes first (fewer spinning instructions); at most `tries`.
__device__ __forceinline__ bool nn_mbar_wait(uint64_t* bar, unsigned parity, int tries = 1 << 20) {
    const uint32_t a = sm_u32(bar);
    for (int it = 0; it < tries; ++it) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(a), "r"(parity), "r"(2000u)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
struct ConvArgs {
    const __nv_bfloat16* x; // [V][cin]
    const __nv_bfloat16* w; // [cout][27][cin]
    const float* bias;      // [cout] or null
    void* y;                // [V][cout], BF16 or FP32
    const __nv_bfloat16* mask; // [V][cout] or null: y *= (mask > 0)
    int nx, ny, nz, cin, cout;
    int relu, y_f32;
    int* err; // set when an mbarrier wait gives up
};

__host__ __device__ constexpr uint32_t tmem_cols(int cout) {
    return cout <= 32 ? 32u : cout <= 64 ? 64u : cout <= 128 ? 128u : cout <= 256 ? 256u : 512u;
}

// ---- conv3d_brick_kernel ----
// A CTA owns a brick of A UMMA M-tiles (8 x 16 voxels each, side by side in x) and marches it through a z
// range.  Producer warps stage each input plane of the brick plus a one-voxel halo into a ring of plane
// slots with cp.async (zero fill outside the grid), one region per 8-channel group so that every (dy, dx)
// tap's A operand is the same K-major canonical layout at a shifted start address: rows of 8 voxels along
// x at 16 bytes, 8-row groups (y) a halo row apart, the two channel halves of a 16-channel K step one
// region apart.  The weights of all 27 taps stay in shared memory.
// A plane p is read once: it contributes to the output planes p-1, p and p+1, whose accumulators lie side
// by side in TMEM (a ring of four planes), so one product per (dy, dx), K step and tile has N = 3 coutp columns,
// the weights of dz = +1, 0, -1 (two products where the ring wraps).  A product reads a 4 KB A tile whatever
// N is and takes about 70 cycles with 16 columns, 100 with 48.  One warp issues them; four epilogue
// warps drain an output plane that is complete (bias, ReLU or mask, BF16 / FP32 store) and clear it for the
// plane that takes its place, while the products of the next plane run.  Every wait is bounded.
// 16 -> 16 channels at 128^3: 0.145 ms with one product per tap and plane -> 0.101 ms; 48 -> 16: 0.442 -> 0.259 ms;
// 128 -> 64 at 32^3: 0.310 ms when its taps were gathered into shared memory -> 0.111 ms in four launches.
constexpr int BR_MAXNP = 8;                    // input plane slots, at most
constexpr int BR_OUT = 4;                      // output planes in TMEM: three in work, one being drained
constexpr int BR_PROD = 4, BR_EPI = 4;         // producer and epilogue warps
constexpr int BR_NT = (BR_PROD + 1 + BR_EPI) * 32;
// Brick geometry: A UMMA M-tiles of 8 x 16 voxels side by side in x (brick 8A x 16), a ring of
// NP input plane slots, each (8A + 2) x 18 voxels x cin channels, one region per 8 channels.
__host__ __device__ constexpr int brick_region(int A) { return (8 * A + 2) * 18 * 16; }
__host__ __device__ constexpr size_t brick_slot_bytes(int A, int cin) { return (size_t)brick_region(A) * (cin / 8); }
__host__ __device__ constexpr size_t brick_smem(int A, int NP, int cin, int coutp) {
    return (size_t)27 * coutp * cin * 2 + NP * brick_slot_bytes(A, cin) + 256;
}
__host__ __device__ constexpr uint32_t brick_tmem_cols(int A, int coutp) { return tmem_cols(BR_OUT * A * coutp); }

// K-major descriptor with explicit leading / stride byte offsets
__device__ __forceinline__ uint64_t kdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void nn_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sm_u32(bar)) : "memory");
}

struct BrickArgs {
    int A, NP;        // M-tiles per brick row, input plane slots
    int co0, coutp;   // the output channels [co0, co0 + coutp) of a.cout computed by this launch
    int zchunk;       // planes per brick
};

template <int A>
__global__ void __launch_bounds__(BR_NT, 1) conv3d_brick_kernel(const ConvArgs a, const BrickArgs g) {
    extern __shared__ __align__(1024) unsigned char br_sm[];
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int cin = a.cin, ctot = a.cout, nhg = cin / 8;
    const int NP = g.NP, co0 = g.co0, coutp = g.coutp, zchunk = g.zchunk;
    const int W = 8 * A + 2;                       // slot width in voxels
    const int REG = brick_region(A);               // bytes of one 8-channel region
    const size_t SLOT = brick_slot_bytes(A, cin);
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    unsigned char* wsm = br_sm;                                   // weights: [t][hg][coutp] x 16 B
    unsigned char* slots = br_sm + (size_t)27 * coutp * cin * 2;  // NP plane slots
    uint64_t* bars = reinterpret_cast<uint64_t*>(slots + NP * SLOT);
    uint64_t* full = bars;                 // [NP] plane staged (BR_PROD*32 arrivals)
    uint64_t* empty = bars + BR_MAXNP;     // [NP] plane no longer read (MMA commit)
    uint64_t* tfull = bars + 2 * BR_MAXNP; // [BR_OUT] output plane complete (MMA commit)
    uint64_t* tempty = tfull + BR_OUT;     // [BR_OUT] output plane drained and cleared (BR_EPI*32 arrivals)
    uint64_t* drain = tempty + BR_OUT;     // [1] every MMA of the CTA done (teardown)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    int* s_fail = reinterpret_cast<int*>(tmem_slot + 1);
    const uint32_t ncols = brick_tmem_cols(A, coutp);
    const int mma_warp = BR_PROD;

    // weights of every tap (output channels co0..) in the canonical B layout: rows at 16 B, 8-row groups
    // 128 B apart; per (dy, dx) and 8 input channels a region of 3 coutp rows, dz = +1, 0, -1
    for (int q = tid; q < 27 * coutp * nhg; q += BR_NT) {
        const int t = q / (coutp * nhg), r = q % (coutp * nhg), n = r / nhg, hg = r % nhg;
        cp_async16(sm_u32(wsm) + (uint32_t)(((((t % 9) * nhg + hg) * 3 + 2 - t / 9) * coutp + n) * 16),
                   a.w + ((size_t)(co0 + n) * 27 + t) * cin + hg * 8, true);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (warp == mma_warp) {
        tmem_alloc(tmem_slot, ncols);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < NP; ++i) {
            nn_mbar_init(&full[i], BR_PROD * 32);
            nn_mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < BR_OUT; ++i) {
            nn_mbar_init(&tfull[i], 1);
            nn_mbar_init(&tempty[i], BR_EPI * 32);
        }
        nn_mbar_init(drain, 1);
        *s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // weights -> tensor core
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp > mma_warp) { // every output plane starts at zero
        for (int c0 = 0; c0 < BR_OUT * A * coutp; c0 += 16)
            tmem_zero16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0);
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const int bw = 8 * A;
    const int bx = (nx + bw - 1) / bw, by = (ny + 15) / 16, nzc = (nz + zchunk - 1) / zchunk;
    const int nbricks = bx * by * nzc;
    bool fail = false;

    if (warp < BR_PROD) {
        // ---------------- producers: the brick's input planes, in order ----------------
        // The copies of plane p are committed as one group; the previous plane's group is then
        // waited for, fenced towards the tensor core's proxy and announced, so that one plane's
        // copies are always in flight while the previous one is published.
        unsigned pc = 0;          // planes staged so far (ring position)
        const int K = min(NP - 1, 5); // planes whose copies stay in flight (one slot is being read)
        int pend[BR_MAXNP] = {}, np_ = 0, ph = 0; // committed, not yet announced slots (oldest at ph)
        const uint32_t inv_h = (65536u + nhg - 1) / nhg; // q / nhg by a multiply, exact for q < 4096
        // wait until at most n copy groups of this thread are pending
        auto wait_groups = [](int n) {
            switch (n) {
            case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
            case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
            case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
            case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
            case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
            default: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
            }
        };
        // announce the oldest pending plane once its copies have landed
        auto publish_oldest = [&]() {
            wait_groups(np_ - 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic -> async proxy
            nn_mbar_arrive(&full[pend[ph]]);
            ph = (ph + 1) % BR_MAXNP;
            --np_;
        };
        for (int br = blockIdx.x; br < nbricks && !fail; br += gridDim.x) {
            const int col = br % (bx * by), zc = br / (bx * by);
            const int x0 = (col % bx) * bw, y0 = (col / bx) * 16;
            const int z0 = zc * zchunk, z1 = min(nz, z0 + zchunk);
            for (int p = z0 - 1; p <= z1 && !fail; ++p, ++pc) {
                const int sl = (int)(pc % NP);
                if (pc >= (unsigned)NP) { // one lane per warp waits for the slot, the warp follows
                    bool ok = lane == 0 ? nn_mbar_wait(&empty[sl], ((pc / NP) - 1) & 1u) : true;
                    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                    if (!ok) {
                        fail = true;
                        break;
                    }
                }
                const uint32_t base = sm_u32(slots + (size_t)sl * SLOT);
                const bool pin = p >= 0 && p < nz;
                // a warp takes a row of voxels at a time, lanes along (voxel, 8 channels): a row
                // is read as consecutive 16-byte pieces
                for (int yy = warp; yy < 18; yy += BR_PROD) {
                    const int gy = y0 - 1 + yy;
                    const bool rin = pin && gy >= 0 && gy < ny;
                    const __nv_bfloat16* row = a.x + ((long long)(rin ? p : 0) * ny + (rin ? gy : 0)) * nx * cin;
                    const uint32_t dst = base + (uint32_t)(yy * W * 16);
                    for (int q = lane; q < W * nhg; q += 32) {
                        const int xx = (int)((q * inv_h) >> 16), hg = q - xx * nhg, gx = x0 - 1 + xx;
                        const bool ok = rin && gx >= 0 && gx < nx;
                        cp_async16(dst + (uint32_t)(hg * REG + xx * 16), ok ? row + (long long)gx * cin + hg * 8 : a.x, ok);
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                pend[(ph + np_) % BR_MAXNP] = sl;
                ++np_;
                while (np_ > K) publish_oldest();
            }
        }
        while (np_ > 0) publish_oldest(); // the last planes
        if (fail) atomicExch(s_fail, 1);
    } else if (warp == mma_warp) {
        // ---------------- MMA issuer (one warp, its elected lane issues) ----------------
        const uint32_t leader = elect_one();
        const uint64_t bbase = kdesc(sm_u32(wsm), (uint32_t)(3 * coutp * 16), 128u);
        const uint32_t bhi = (uint32_t)(bbase >> 32), tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
        unsigned pc = 0, on = 0; // planes waited for, output planes of the bricks before this one
        for (int br = blockIdx.x; br < nbricks && !fail; br += gridDim.x) {
            const int zc = br / (bx * by);
            const int z0 = zc * zchunk, z1 = min(nz, z0 + zchunk);
            for (int p = z0 - 1; p <= z1 && !fail; ++p, ++pc) {
                if (!__all_sync(0xffffffffu, nn_mbar_wait(&full[pc % NP], (pc / NP) & 1u))) {
                    fail = true;
                    break;
                }
                // the output planes that p contributes to; p + 1 is new: its place must be cleared
                const int zlo = max(z0, p - 1), zhi = min(z1 - 1, p + 1);
                const unsigned olo = on + (unsigned)(zlo - z0), ohi = on + (unsigned)(zhi - z0);
                if (zhi == p + 1 && ohi >= (unsigned)BR_OUT &&
                    !__all_sync(0xffffffffu, nn_mbar_wait(&tempty[ohi % BR_OUT], (ohi / BR_OUT - 1) & 1u))) {
                    fail = true;
                    break;
                }
                tc_fence_after();
                const uint64_t abase = kdesc(sm_u32(slots + (size_t)(pc % NP) * SLOT), (uint32_t)REG, (uint32_t)(W * 16));
                const uint32_t ahi = (uint32_t)(abase >> 32);
                // runs of output planes at consecutive places of the ring
                for (unsigned o = olo; o <= ohi;) {
                    const unsigned cnt = min(ohi - o + 1, (unsigned)BR_OUT - o % BR_OUT);
                    const int blk = (int)(o - olo) + zlo - (p - 1); // first weight block (dz = +1, 0, -1)
                    const uint32_t idesc = idesc_bf16(CONV_TM, (int)cnt * coutp);
                    const uint32_t dacc = tmem_u + (o % BR_OUT) * (uint32_t)coutp;
                    for (int s2 = 0; s2 < cin / 16; ++s2) {
                        const uint32_t a_s = (uint32_t)abase + (uint32_t)(2 * s2 * (REG >> 4));
                        const uint32_t b_s = (uint32_t)bbase + (uint32_t)((2 * s2 * 3 + blk) * coutp);
#pragma unroll
                        for (int tyx = 0; tyx < 9; ++tyx) {
                            const int dy = tyx / 3, dx = tyx % 3; // 0..2: offsets + 1
                            const uint32_t bd = b_s + (uint32_t)(tyx * nhg * 3 * coutp);
#pragma unroll
                            for (int j = 0; j < A; ++j)
                                umma_bf16_warp(dacc + (uint32_t)(j * BR_OUT * coutp), a_s + (uint32_t)(dy * W + dx + 8 * j),
                                               ahi, bd, bhi, idesc, 1u, leader);
                        }
                    }
                    o += cnt;
                }
                umma_commit_warp(&empty[pc % NP], leader);
                if (p > z0) umma_commit_warp(&tfull[(on + (unsigned)(p - 1 - z0)) % BR_OUT], leader); // plane p - 1
            }
            on += (unsigned)(z1 - z0);
        }
        if (fail && lane == 0) atomicExch(s_fail, 1);
    } else {
        // ---------------- epilogue warps: TMEM -> registers -> global ----------------
        const int q = warp & 3;      // TMEM lane quarter this warp may access
        const int m = q * 32 + lane; // row of an M-tile: x = m % 8, y = m / 8
        unsigned pw = 0;
        for (int br = blockIdx.x; br < nbricks && !fail; br += gridDim.x) {
            const int col = br % (bx * by), zc = br / (bx * by);
            const int x0 = (col % bx) * bw, y0 = (col / bx) * 16;
            const int z0 = zc * zchunk, z1 = min(nz, z0 + zchunk);
            for (int z = z0; z < z1 && !fail; ++z, ++pw) {
                const int tb = (int)(pw % BR_OUT);
                // one lane waits, the warp follows (the TMEM loads below are warp-collective)
                bool ok = lane == 0 ? nn_mbar_wait(&tfull[tb], (pw / BR_OUT) & 1u) : true;
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) {
                    fail = true;
                    break;
                }
                tc_fence_after();
                for (int j = 0; j < A; ++j) {
                    const int gx = x0 + 8 * j + (m & 7), gy = y0 + (m >> 3);
                    const bool vin = gx < nx && gy < ny;
                    const size_t v = ((size_t)z * ny + gy) * nx + gx;
                    for (int c0 = 0; c0 < coutp; c0 += 16) {
                        float acc[16];
                        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((j * BR_OUT + tb) * coutp + c0);
                        __syncwarp(); // (the loads are warp-collective)
                        tmem_ld16(at, acc);
                        tmem_zero16(at);
                        if (!vin) continue;
                        const int cg = co0 + c0; // channel in the full output
                        if (a.bias)
#pragma unroll
                            for (int i = 0; i < 16; ++i) acc[i] += __ldg(a.bias + cg + i);
                        if (a.relu)
#pragma unroll
                            for (int i = 0; i < 16; ++i) acc[i] = fmaxf(acc[i], 0.f);
                        if (a.mask) {
                            const uint4* mp = reinterpret_cast<const uint4*>(a.mask + v * ctot + cg);
                            const uint4 m0 = __ldg(mp), m1 = __ldg(mp + 1);
                            const __nv_bfloat16* mb0 = reinterpret_cast<const __nv_bfloat16*>(&m0);
                            const __nv_bfloat16* mb1 = reinterpret_cast<const __nv_bfloat16*>(&m1);
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                if (!(__bfloat162float(mb0[i]) > 0.f)) acc[i] = 0.f;
                                if (!(__bfloat162float(mb1[i]) > 0.f)) acc[8 + i] = 0.f;
                            }
                        }
                        if (a.y_f32) {
                            float4* yp = reinterpret_cast<float4*>(static_cast<float*>(a.y) + v * ctot + cg);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                yp[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
                        } else {
                            __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                            for (int i = 0; i < 16; ++i) o[i] = __float2bfloat16(acc[i]);
                            uint4* yp = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.y) + v * ctot + cg);
                            yp[0] = reinterpret_cast<const uint4*>(o)[0];
                            yp[1] = reinterpret_cast<const uint4*>(o)[1];
                        }
                    }
                }
                __syncwarp();
                tmem_wait_st();
                tc_fence_before();
                nn_mbar_arrive(&tempty[tb]);
            }
        }
        if (fail) atomicExch(s_fail, 1);
    }
    // ---- teardown: every role has stopped issuing; the MMAs still in flight are waited for
    // (one more commit tracks all of them) before the accumulator is released ----
    __syncthreads();
    if (warp == mma_warp) { // (the lane that issued them commits)
        umma_commit_warp(drain, elect_one());
        if (!nn_mbar_wait(drain, 0u)) atomicExch(s_fail, 1);
    }
    __syncthreads();
    if (*s_fail && tid == 0) atomicExch(a.err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == mma_warp) {
        tc_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// ---- weight gradient: dW[co][t][ci] = sum_v dY[v][co] X[v + off(t)][ci] ----
// A contraction over the voxels (K), so both operands are read channel-major ("MN-major") and
// the activations need no transposition: in a staged plane, one region per 8 channels with a
// voxel's 16 bytes at consecutive addresses, 8 consecutive voxels are one core matrix.
//   M = 128 rows: 16 consecutive 8-channel regions of X, which run over the channels of a plane
//     and then over the next planes; the dz taps of a voxel plane are 3 planes, so one product
//     covers all three (and, with Q voxel planes in N, all Q + 2).  Rows past them are unused.
//   N = Q * coN columns: the output channels of Q consecutive voxel planes of dY.
//   K = 16 voxels along x; the dy and dx taps are shifted start addresses of X.
// The Q voxel planes' blocks of the result are separate partial sums (row plane p and column
// plane q belong to tap dz = p - q).  A CTA walks voxel bricks (16 x BY x BZ, two in flight where
// shared memory allows) with an accumulator per (dy, dx) and M tile in TMEM.  The tensor core truncates
// when it adds to an accumulator, and a chain of n products loses about 1.3e-8 n of its sum (measured:
// 304 products 4.0e-6, 913 products 1.4e-5), so after every BY products the accumulators are added to
// 32-bit sums in registers (rounded to nearest) and start again at zero: 8e-8 over 128^3 voxels,
// against 1.1e-7 for chains of 32-bit multiply-adds.
// Each CTA's sums go to part[chunk * Q + q] and wgrad_reduce_kernel adds those in a fixed order.  The bias
// gradient is summed from the staged dY on the CUDA cores while the tensor core runs.
// Bound by the products (an A tile of 4 KB each, 90 to 140 cycles at 16 to 32 columns).  The twelve layers of
// a 128^3 sample: 2.1 ms, against 29.6 ms as FP32 register tiles on the CUDA cores (and 1.3 ms for
// their bias gradients, which are now part of it); 16 -> 16 channels at 128^3: 0.29 ms.
constexpr int WG_NT = 512;
constexpr int WG_COLS = 320; // accumulator columns, at most: 5 groups of 16 per warp, 80 registers
constexpr int WG_BX = 16, WG_XW = WG_BX + 2;
struct WgArgs {
    const __nv_bfloat16* x;  // [V][cin]
    const __nv_bfloat16* dy; // [V][cout]
    float* part;             // [nchunks * Q][cout][27][cin]
    float* bpart;            // [nchunks][cout]
    int nx, ny, nz, cin, cout;
    int Q, tiles, coN; // voxel planes in N, M tiles, output channels per CTA
    int BY, BZ, stages;     // brick rows and planes (BZ a multiple of Q), bricks staged at a time
    int* err;               // set when an mbarrier wait gives up
};
__host__ __device__ constexpr int wg_xreg(int BY) { return WG_XW * (BY + 2) * 16; } // one 8-channel region of a plane
__host__ __device__ constexpr int wg_yreg(int BY) { return WG_BX * BY * 16; }
__host__ __device__ constexpr size_t wg_xbytes(int cin, int BY, int BZ) {
    return (size_t)(BZ + 2) * (cin / 8) * wg_xreg(BY);
}
__host__ __device__ constexpr size_t wg_ybytes(int coN, int BY, int BZ) {
    return (size_t)BZ * (coN / 8) * wg_yreg(BY);
}
// shared memory of a launch: the bricks, and what the unused rows of the last one read past it
constexpr size_t wg_smem(int cin, int coN, int Q, int tiles, int BY, int BZ, int stages) {
    const long long xb = (long long)wg_xbytes(cin, BY, BZ), yb = (long long)wg_ybytes(coN, BY, BZ);
    const long long over = (16ll * tiles - (long long)(Q + 2) * (cin / 8)) * wg_xreg(BY);
    return (size_t)((stages - 1) * (xb + yb) + xb + (over > yb ? over : yb));
}

template <int NDT>
__global__ void __launch_bounds__(WG_NT, 1) wgrad_tc_kernel(const WgArgs a) {
    extern __shared__ __align__(1024) unsigned char wg_sm[];
    __shared__ __align__(8) uint64_t bar; // the products issued last have completed
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int cin = a.cin, cout = a.cout, nhg = cin / 8, coN = a.coN, nho = coN / 8, Q = a.Q, tiles = a.tiles;
    const int BY = a.BY, BZ = a.BZ, stages = a.stages;
    constexpr int ndt = NDT; // 9: every (dy, dx); 3: dy = blockIdx.y, every dx
    const int co0 = blockIdx.z * coN, td0 = blockIdx.y * ndt;
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int XREG = wg_xreg(BY), YREG = wg_yreg(BY);
    const uint32_t xbytes = (uint32_t)wg_xbytes(cin, BY, BZ), sbytes = xbytes + (uint32_t)wg_ybytes(coN, BY, BZ);
    const uint32_t base = sm_u32(wg_sm);
    const int ncol = Q * coN;
    const uint32_t ncols = tmem_cols(ndt * tiles * ncol);
    if (warp == 0) {
        tmem_alloc(&tmem_slot, ncols);
        tmem_relinquish();
    }
    if (tid == 0) {
        nn_mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, tmem_u = __shfl_sync(0xffffffffu, tmem, 0), leader = elect_one();
    const int nbx = (nx + WG_BX - 1) / WG_BX, nby = (ny + BY - 1) / BY, nbz = (nz + BZ - 1) / BZ;
    const int nblk = nbx * nby * nbz;

    // copies of one brick: a warp takes a row of voxels at a time, lanes along (voxel, 8 channels),
    // so that a row is read as consecutive 16-byte pieces; zeros outside the grid
    const uint32_t inv_h = (65536u + nhg - 1) / nhg, inv_o = (65536u + nho - 1) / nho; // exact for < 4096
    auto load = [&](int b, int buf) {
        const int x0 = (b % nbx) * WG_BX, y0 = ((b / nbx) % nby) * BY, z0 = (b / (nbx * nby)) * BZ;
        const uint32_t xs = base + buf * sbytes, ys = xs + xbytes;
        const int xrows = (BZ + 2) * (BY + 2), xlen = WG_XW * nhg;
        for (int r = warp; r < xrows; r += WG_NT / 32) {
            const int pz = r / (BY + 2), yy = r - pz * (BY + 2);
            const int gz = z0 + pz - 1, gy = y0 + yy - 1;
            const bool rin = gz >= 0 && gz < nz && gy >= 0 && gy < ny;
            const __nv_bfloat16* row = a.x + ((long long)(rin ? gz : 0) * ny + (rin ? gy : 0)) * nx * cin;
            const uint32_t dst = xs + (uint32_t)(pz * nhg * XREG + yy * (WG_XW * 16));
            for (int q = lane; q < xlen; q += 32) {
                const int xx = (int)((q * inv_h) >> 16), hg = q - xx * nhg, gx = x0 + xx - 1;
                const bool ok = rin && gx >= 0 && gx < nx;
                cp_async16(dst + (uint32_t)(hg * XREG + xx * 16), ok ? row + (long long)gx * cin + hg * 8 : a.x, ok);
            }
        }
        const int yrows = BZ * BY, ylen = WG_BX * nho;
        for (int r = warp; r < yrows; r += WG_NT / 32) {
            const int pz = r / BY, yy = r - pz * BY;
            const int gz = z0 + pz, gy = y0 + yy;
            const bool rin = gz < nz && gy < ny;
            const __nv_bfloat16* row = a.dy + ((long long)(rin ? gz : 0) * ny + (rin ? gy : 0)) * nx * cout + co0;
            const uint32_t dst = ys + (uint32_t)(pz * nho * YREG + yy * (WG_BX * 16));
            for (int q = lane; q < ylen; q += 32) {
                const int xx = (int)((q * inv_o) >> 16), hg = q - xx * nho, gx = x0 + xx;
                const bool ok = rin && gx < nx;
                cp_async16(dst + (uint32_t)(hg * YREG + xx * 16), ok ? row + (long long)gx * cout + hg * 8 : a.dy, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // bias gradient: a thread sums one 8-channel group over a strided share of the brick's voxels
    const bool bias = blockIdx.y == 0;
    int per = WG_NT / 2; // threads per group, a power of two
    while (per * nho > WG_NT) per >>= 1;
    const int bhg = tid / per, bsub = tid % per;
    float bacc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) bacc[i] = 0.f;

    const uint32_t idesc = idesc_bf16(CONV_TM, ncol) | (1u << 15) | (1u << 16); // A and B MN-major
    // this warp's accumulator columns: groups of 16, every 4th (four warps share a lane quarter)
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int groups = ndt * tiles * (ncol / 16);
    constexpr int GW = WG_COLS / 64;
    float sum[GW][16];
#pragma unroll
    for (int e = 0; e < GW; ++e)
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[e][i] = 0.f;
    unsigned phase = 0u;
    bool fail = false;
    if ((int)blockIdx.x < nblk) load(blockIdx.x, 0);
    int buf = 0;
    for (int b = blockIdx.x; b < nblk && !fail; b += gridDim.x) {
        const int bn = b + gridDim.x;
        const bool ahead = stages == 2 && bn < nblk;
        if (ahead) { // (the other buffer was left before the last barrier)
            load(bn, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        const uint32_t xs = base + buf * sbytes, ys = xs + xbytes;
        const uint64_t ad0 = kdesc(xs, 128u, (uint32_t)XREG), bd0 = kdesc(ys, 128u, (uint32_t)YREG);
        const uint32_t ahi = (uint32_t)(ad0 >> 32), bhi = (uint32_t)(bd0 >> 32);
        const uint32_t a0 = (uint32_t)ad0 + (NDT == 9 ? 0u : (uint32_t)(blockIdx.y * WG_XW));
        for (int zq = 0; zq < BZ; zq += Q) {
            if (warp == 0) {
                tc_fence_after();
                for (int y = 0; y < BY; ++y) {
                    const uint32_t bd = (uint32_t)bd0 + (uint32_t)((zq * nho * YREG + y * (WG_BX * 16)) >> 4);
                    const uint32_t ay = a0 + (uint32_t)((zq * nhg * XREG) >> 4) + (uint32_t)(y * WG_XW);
                    for (int tl = 0; tl < tiles; ++tl)
#pragma unroll
                        for (int d = 0; d < NDT; ++d) // (dy, dx) = (d / 3, d % 3), offsets + 1
                            umma_bf16_warp(tmem_u + (uint32_t)((d * tiles + tl) * ncol),
                                           ay + (uint32_t)(tl * XREG) + (uint32_t)((d / 3) * WG_XW + d % 3), ahi, bd, bhi,
                                           idesc, y > 0 ? 1u : 0u, leader);
                }
                umma_commit_warp(&bar, leader);
            }
            if (bias && bhg < nho) { // the bias gradient's share of these planes, meanwhile
                const unsigned char* yb = wg_sm + buf * sbytes + xbytes;
                for (int z = zq; z < zq + Q; ++z) {
                    const uint4* row = reinterpret_cast<const uint4*>(yb + (size_t)(z * nho + bhg) * YREG);
                    for (int v = bsub; v < WG_BX * BY; v += per) {
                        const uint4 raw = row[v];
                        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
                        for (int i = 0; i < 8; ++i) bacc[i] += __bfloat162float(e[i]);
                    }
                }
            }
            __syncwarp();
            if (!nn_mbar_wait(&bar, phase)) fail = true;
            phase ^= 1u;
            tc_fence_after();
            if (!__any_sync(0xffffffffu, fail)) {
#pragma unroll
                for (int e = 0; e < GW; ++e) {
                    const int g = (warp >> 2) + 4 * e;
                    if (g < groups) { // (warp-uniform)
                        float v[16];
                        tmem_ld16(lane_base + (uint32_t)(g * 16), v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[e][i] += v[i];
                    }
                }
            }
            tc_fence_before();
            // the accumulators are read (and, after the last planes, the buffer is left)
            fail = __syncthreads_or(fail);
            if (fail) break;
        }
        if (stages == 1 && bn < nblk && !fail) load(bn, 0);
        if (stages == 2) buf ^= 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!fail) {
        const int m = (warp & 3) * 32 + lane;
#pragma unroll
        for (int e = 0; e < GW; ++e) {
            const int gi = (warp >> 2) + 4 * e;
            if (gi >= groups) break;
            const int dt = gi / (ncol / 16), c0 = (gi % (ncol / 16)) * 16;
            const int d = dt / tiles, tl = dt % tiles;
            const int g = 16 * tl + (m >> 3), qq = c0 / coN, dz = g / nhg - qq;
            if (dz >= 0 && dz <= 2) {
                const int ci = (g % nhg) * 8 + (m & 7), t = dz * 9 + td0 + d, co = co0 + c0 - qq * coN;
                float* o = a.part + (((size_t)blockIdx.x * Q + qq) * cout + co) * 27 * cin + (size_t)t * cin + ci;
#pragma unroll
                for (int i = 0; i < 16; ++i) o[(size_t)i * 27 * cin] = sum[e][i];
            }
        }
        if (bias) { // lanes of one channel group, then the warps, in index order
            float(*bred)[CONV_MAXC] = reinterpret_cast<float(*)[CONV_MAXC]>(wg_sm); // (the bricks are done with)
            for (int w = tid; w < (WG_NT / 32) * CONV_MAXC; w += WG_NT) bred[w / CONV_MAXC][w % CONV_MAXC] = 0.f;
            __syncthreads();
            // a warp may hold the lanes of several channel groups (per < 32)
            const int span = per < 32 ? per : 32;
            for (int o = span >> 1; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float other = __shfl_down_sync(0xffffffffu, bacc[i], o);
                    if ((lane & (span - 1)) + o < span) bacc[i] += other;
                }
            if (bhg < nho && (lane & (span - 1)) == 0)
#pragma unroll
                for (int i = 0; i < 8; ++i) bred[warp][bhg * 8 + i] = bacc[i];
            __syncthreads();
            for (int c = tid; c < coN; c += WG_NT) {
                float s = 0.f;
                for (int w = 0; w < WG_NT / 32; ++w) s += bred[w][c];
                a.bpart[(size_t)blockIdx.x * cout + co0 + c] = s;
            }
        }
    } else if (tid == 0) {
        atomicExch(a.err, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// dw (+)= sum over np partials of n values, db (+)= sum over nb partials of m values: 32 values
// per block, 8 threads a value, each over every 8th partial, then the 8 in order (deterministic)
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ part, int np, size_t n,
                                                           float* __restrict__ dw, const float* __restrict__ bpart,
                                                           int nb, int m, float* __restrict__ db, int accumulate) {
    __shared__ float red[8][33];
    const size_t nblk = (n + 31) / 32;
    const bool w = blockIdx.x < nblk;
    const size_t e = (w ? (size_t)blockIdx.x : (size_t)blockIdx.x - nblk) * 32 + threadIdx.x, len = w ? n : (size_t)m;
    const float* src = w ? part : bpart;
    float* dst = w ? dw : db;
    const int cnt = w ? np : nb;
    float s = 0.f;
    if (e < len) {
#pragma unroll 4
        for (int c = threadIdx.y; c < cnt; c += 8) s += src[(size_t)c * len + e];
    }
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && e < len) {
#pragma unroll
        for (int k = 1; k < 8; ++k) s += red[k][threadIdx.x];
        dst[e] = accumulate ? dst[e] + s : s;
    }
}

// W'[ci][t][co] = W[co][26 - t][ci]: the data gradient as a forward convolution
__global__ void flip_weights_kernel(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt, int cin,
                                    int cout) {
    const int n = cout * 27 * cin;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int co = e / (27 * cin), t = (e / cin) % 27, ci = e % cin;
        wt[((size_t)ci * 27 + (26 - t)) * cout + co] = w[e];
    }
}

// ---- pooling, upsampling with concatenation, and their gradients (C channels) ----
// (8 channels per thread in all of them: 16-byte accesses)
struct Bf8 {
    float f[8];
};
__device__ __forceinline__ Bf8 bf8_load(const __nv_bfloat16* p) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(p));
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
    Bf8 v;
#pragma unroll
    for (int i = 0; i < 8; ++i) v.f[i] = __bfloat162float(e[i]);
    return v;
}
__device__ __forceinline__ void bf8_store(__nv_bfloat16* p, const Bf8& v) {
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = __float2bfloat16(v.f[i]);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(o);
}
// average of the 8 children; fine grid (nx, ny, nz) even
__global__ void pool_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int nx, int ny,
                            int nz, int C) {
    const int cx = nx / 2, cy = ny / 2, cz = nz / 2, Q = C / 8;
    const size_t n = (size_t)cx * cy * cz * Q;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int q = (int)(e % Q);
        const size_t P = e / Q;
        const int I = (int)(P % cx), J = (int)((P / cx) % cy), K = (int)(P / ((size_t)cx * cy));
        Bf8 s{};
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            const int i = 2 * I + (d & 1), j = 2 * J + ((d >> 1) & 1), k = 2 * K + (d >> 2);
            const Bf8 v = bf8_load(x + ((size_t)i + (size_t)nx * ((size_t)j + (size_t)ny * k)) * C + 8 * q);
#pragma unroll
            for (int u = 0; u < 8; ++u) s.f[u] += v.f[u];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) s.f[u] *= 0.125f;
        bf8_store(y + P * C + 8 * q, s);
    }
}
// Gradient of an encoder level's output from its two uses, times its ReLU derivative:
// g[v] = (skip[v] + dy[parent] / 8) where act[v] > 0, summed in FP32
__global__ void skip_pool_bwd_kernel(const __nv_bfloat16* __restrict__ skip, const __nv_bfloat16* __restrict__ dy,
                                     const __nv_bfloat16* __restrict__ act, __nv_bfloat16* __restrict__ g, int nx,
                                     int ny, int nz, int C) {
    const int cx = nx / 2, cy = ny / 2, Q = C / 8;
    const size_t n = (size_t)nx * ny * nz * Q;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int q = (int)(e % Q);
        const size_t v = e / Q;
        const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((size_t)nx * ny));
        const size_t P = (size_t)(i >> 1) + (size_t)cx * ((size_t)(j >> 1) + (size_t)cy * (k >> 1));
        const Bf8 s = bf8_load(skip + v * C + 8 * q), d = bf8_load(dy + P * C + 8 * q), a = bf8_load(act + v * C + 8 * q);
        Bf8 o;
#pragma unroll
        for (int u = 0; u < 8; ++u) o.f[u] = a.f[u] > 0.f ? s.f[u] + 0.125f * d.f[u] : 0.f;
        bf8_store(g + v * C + 8 * q, o);
    }
}
// cat[v] = (coarse[parent(v)] (Ca channels), skip[v] (Cb channels)); fine grid (nx, ny, nz);
// one thread per 8-channel chunk (Ca, Cb multiples of 8)
__global__ void upcat_kernel(const __nv_bfloat16* __restrict__ coarse, const __nv_bfloat16* __restrict__ skip,
                             __nv_bfloat16* __restrict__ cat, int nx, int ny, int nz, int Ca, int Cb) {
    const int qa = Ca / 8, qb = Cb / 8, Q = qa + qb, cx = nx / 2, cy = ny / 2;
    const size_t n = (size_t)nx * ny * nz * Q;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int q = (int)(e % Q);
        const size_t v = e / Q;
        uint4 val;
        if (q < qa) {
            const int i = (int)(v % nx);
            const size_t r = v / nx;
            const int j = (int)(r % ny), k = (int)(r / ny);
            const size_t P = (size_t)(i >> 1) + (size_t)cx * ((size_t)(j >> 1) + (size_t)cy * (k >> 1));
            val = __ldg(reinterpret_cast<const uint4*>(coarse + P * Ca) + q);
        } else {
            val = __ldg(reinterpret_cast<const uint4*>(skip + v * Cb) + (q - qa));
        }
        reinterpret_cast<uint4*>(cat + v * (Ca + Cb))[q] = val;
    }
}
// Gradient of upcat: g[P] = (sum over the 8 children of dcat[child][0:Ca]) where act[P] > 0 (the ReLU derivative of
// the coarse activation; FP32 sum), and skip[v] = dcat[v][Ca:], kept for the encoder.  One thread per coarse
// cell and 8 channels of dcat: dcat is read once.
__global__ void upcat_bwd_kernel(const __nv_bfloat16* __restrict__ dcat, const __nv_bfloat16* __restrict__ act,
                                 __nv_bfloat16* __restrict__ g, __nv_bfloat16* __restrict__ skip, int nx, int ny,
                                 int nz, int Ca, int Cb) {
    const int C = Ca + Cb, cx = nx / 2, cy = ny / 2, cz = nz / 2, Q = C / 8, qa = Ca / 8;
    const size_t n = (size_t)cx * cy * cz * Q;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int q = (int)(e % Q);
        const size_t P = e / Q;
        const int I = (int)(P % cx), J = (int)((P / cx) % cy), K = (int)(P / ((size_t)cx * cy));
        auto child = [&](int d) {
            const int i = 2 * I + (d & 1), j = 2 * J + ((d >> 1) & 1), k = 2 * K + (d >> 2);
            return (size_t)i + (size_t)nx * ((size_t)j + (size_t)ny * k);
        };
        if (q < qa) {
            Bf8 s{};
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                const Bf8 v = bf8_load(dcat + child(d) * C + 8 * q);
#pragma unroll
                for (int u = 0; u < 8; ++u) s.f[u] += v.f[u];
            }
            const Bf8 a = bf8_load(act + P * Ca + 8 * q);
#pragma unroll
            for (int u = 0; u < 8; ++u) s.f[u] = a.f[u] > 0.f ? s.f[u] : 0.f;
            bf8_store(g + P * Ca + 8 * q, s);
        } else {
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                const size_t v = child(d);
                *reinterpret_cast<uint4*>(skip + v * Cb + 8 * (q - qa)) = __ldg(reinterpret_cast<const uint4*>(dcat + v * C) + q);
            }
        }
    }
}
// ---- network input, output and loss ----
// input channels: 0 lnK / 2, 1 the x-linear head guess - 1/2 (centred), 2..15 zero.
// h_lin = h_w + (h_e - h_w) (i + 1/2) / nx (init_head_guess, solve_head.cu:56-73)
// from lnK (training data, FP32) or from K (the solver's input, FP64: lnK = log K)
template <class TIN, bool FROM_K>
__global__ void nn_input_kernel(const TIN* __restrict__ src, __nv_bfloat16* __restrict__ in, int nx, int ny, int nz,
                                double hw, double he) {
    const size_t V = (size_t)nx * ny * nz;
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx);
        const double hl = hw + (he - hw) * (i + 0.5) / nx;
        const double lnk = FROM_K ? log((double)src[v]) : (double)src[v];
        __align__(16) __nv_bfloat16 o[16];
        o[0] = __float2bfloat16((float)(0.5 * lnk));
        o[1] = __float2bfloat16((float)(hl - 0.5 * (hw + he)));
        for (int c = 2; c < 16; ++c) o[c] = __float2bfloat16(0.f);
        reinterpret_cast<uint4*>(in + v * 16)[0] = reinterpret_cast<const uint4*>(o)[0];
        reinterpret_cast<uint4*>(in + v * 16)[1] = reinterpret_cast<const uint4*>(o)[1];
    }
}
// x0 = h_lin + scale * out[v][0]
__global__ void nn_output_kernel(const float* __restrict__ out, double* __restrict__ x0, int nx, int ny, int nz,
                                 double hw, double he, double scale) {
    const size_t V = (size_t)nx * ny * nz;
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx);
        const double hl = hw + (he - hw) * (i + 0.5) / nx;
        x0[v] = hl + scale * (double)out[v * 16];
    }
}
// loss = mean over voxels of (out[v][0] - (h - h_lin)/scale)^2; dout (BF16, 16 channels) =
// d loss / d out; per-block partial sums of the squared error in part[blockIdx.x]
__global__ void nn_loss_kernel(const float* __restrict__ out, const float* __restrict__ h,
                               __nv_bfloat16* __restrict__ dout, float* __restrict__ part, int nx, int ny, int nz,
                               double hw, double he, double inv_scale) {
    __shared__ float red[256];
    const size_t V = (size_t)nx * ny * nz;
    float s = 0.f;
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < V; v += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx);
        const double hl = hw + (he - hw) * (i + 0.5) / nx;
        const float target = (float)((h[v] - hl) * inv_scale);
        const float d = out[v * 16] - target;
        s += d * d;
        __align__(16) __nv_bfloat16 o[16];
        o[0] = __float2bfloat16(2.f * d / (float)V);
        for (int c = 1; c < 16; ++c) o[c] = __float2bfloat16(0.f);
        reinterpret_cast<uint4*>(dout + v * 16)[0] = reinterpret_cast<const uint4*>(o)[0];
        reinterpret_cast<uint4*>(dout + v * 16)[1] = reinterpret_cast<const uint4*>(o)[1];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// Adam (Kingma & Ba 2015) on FP32 master weights; the BF16 copy the kernels read is refreshed.
__global__ void adam_kernel(float* __restrict__ w, __nv_bfloat16* __restrict__ wb, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v2, size_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2, float gscale) {
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const float gg = g[e] * gscale;
        const float mm = b1 * m[e] + (1.f - b1) * gg;
        const float vv = b2 * v2[e] + (1.f - b2) * gg * gg;
        m[e] = mm;
        v2[e] = vv;
        const float wn = w[e] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
        w[e] = wn;
        if (wb) wb[e] = __float2bfloat16(wn);
    }
}

} // namespace nn
} // namespace mf3d
