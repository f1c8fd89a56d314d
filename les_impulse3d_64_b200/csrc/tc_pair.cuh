// tc_pair.cuh - the six FDM transforms of the mixed form's pressure pass as three launches of two chained tcgen05
// transforms each (3xTF32, tc_gemm.cuh), for grids whose axes have at most 256 cells.
//
//   forward:  t1[z] = (S_y^T r[z] / rms) S_x            a CTA per z-plane and 128 transformed rows y'
//   z:        t2 = S_z (inv_lambda .* (S_z^T t1))       a CTA per 128 plane columns
//   inverse:  phi[z] += rms (S_y t2[z]) S_x^T           a CTA per z-plane and 128 rows y
//
// Every product has the form D[m][n] = sum_k A[m][k] B[n][k], both operands K-major in shared memory, D in TMEM:
//   forward, inverse:  D1[y'][x] = S_y . field[z]   (A: basis, 128 rows y';  B: field, rows x, k = y)
//                      D2[x'][y'] = S_x . D1        (A: basis, rows x';      B: D1, 128 rows y', k = x)
//   z:                 D1[n][z'] = field . S_z      (A: field, 128 columns n, k = z;  B: basis)
//                      D2[n][z] = (D1 / lambda) . S_z                        (A: D1;  B: basis)
// The first product comes out of TMEM row by row and is split and stored as an operand of the second as it stands: no
// value between the two transforms goes to memory, and no row is transposed.  The field's planes are read, and the
// results written, with a warp's 32 lanes on consecutive elements (that is why the plane launches take y first: with
// x first, and the result's lanes on rows, each 16-byte access of a warp touched 32 lines and the inverse's epilogue
// alone took 16,000 cycles at 128^3).  The split, the three products of a k step and their FP32 accumulation are those
// of the single transforms (tc_gemm.cuh).
//
// Roles: 16 warps bring the field of a 32-wide k panel into registers several panels ahead, two columns per load (8 or
// 16 bytes: a warp's 4-byte loads reach 28 bytes per clock and SM here, 16-byte ones 66), split it into its TF32 hi and
// lo parts and store both in shared memory (first product), then do the same with the first result out of TMEM (second
// product), and write the outcome; one thread copies the basis panels, which are stored split and in shared-memory
// order, with cp.async.bulk; one thread issues the MMAs.  The panels go through a ring of stages, each freed by the
// commit of its MMAs, so copies, splits and MMAs of different panels overlap.  The first basis panels are copied before
// the previous kernel ends (griddepcontrol): they do not depend on it.
//
// Bound: at 128^3, where a launch is one wave of CTAs of 2 x 4 panels, that chain: the first loads, eight panels and the
// stores (18 to 23 us under ncu, tensor pipe 13 to 16% of it, shared-memory data pipe 13 to 18%, most stalls on global
// loads).  With longer rows shared memory: counted at n = 128, a panel's 12 MMAs read 96 KB of operands (768 clocks at 128
// bytes per clock, as long as the MMAs themselves) and 64 KB of splits and copies are written beside them, 1,280 clocks,
// where the same loop took 1,000 to 1,150 with nothing but its MMAs and barriers; at 256 x 256 x 64 the plane launches
// have the tensor pipe busy 27 to 31%.  The inverse holds its potential's values over the products and spills 84 bytes a
// thread (96 registers are what 18 warps leave), the forward launch 48 with rows beyond 128.  A launch at 128^3 took 17 us where its two single launches took 28 (the first passes of a step 250 -> 157 us, the step
// 1.086 -> 0.939 ms); at 164 x 164 x 93 the first passes went from 484 to 370 us, at 256^3 from 2,575 to 1,210 us (the
// step 8.92 -> 6.63 ms).  A pass moves 44 bytes per cell instead of 64.  Splitting the basis here instead (half the
// bytes to copy, twice the splits) measured slower (164 x 164 x 93: 398 us), as did 8 converting warps (417).
// Every wait is bounded (mbar_wait_or_fail): on time-out the kernel records kDeviceWait, waits for its copies and
// MMAs in flight, frees its TMEM and returns.
#pragma once
#include <type_traits>

#include "tc_gemm.cuh"

namespace cavity {

constexpr int kTcPairMax = 256;                 // the largest axis: the two results fill the 512 TMEM columns
constexpr int kTcPairConv = 512;                // threads that split and store (16 warps)
constexpr int kTcPairThreads = kTcPairConv + 64;
constexpr int kTcPairMaxStages = 4;
constexpr int kTcPairPartA = kTcRows * kTcKC * 4;          // bytes of the A panel's hi (or lo) part

enum TcPairMode : int { kTcPairForward = 0, kTcPairZ = 1, kTcPairInverse = 2 };

struct TcPairArgs {
    int nx, ny, nz;
    int n;                         // columns of the first product (nx, or nz for z), rounded up to 32
    int tiles;                     // 128-row tiles of the second product's A (ceil(nx / 128); 1 for z)
    int slot1, stages;             // bytes of a stage's second slot, stages of the ring
    const float *basis1[2], *basis2[2];  // the products' basis images, hi and lo (basis_image_index; r1 and r2 rows)
    int r1, r2;
    const double* r;               // forward: the residual, or
    const double* r_alt;           // the right-hand side when the control block says use_rhs
    const float* in;               // z, inverse
    float* out;                    // forward, z
    const float* inv_lambda;       // z
    double* phi;                   // inverse
    double n_cell;
    const Control* c;
    int* error;
    cudaGraphConditionalHandle handle;
    int clear_condition;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// mbar_wait_bounded for one of several roles: gives up early, and tells the others, when any of them has failed
__device__ __forceinline__ bool mbar_wait_or_fail(uint64_t* bar, uint32_t parity, volatile int* failed) {
    for (long it = 0; it < (1L << 24); it++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 1023) == 1023 && *failed) return false;
    }
    *failed = 1;
    return false;
}
// the same for a whole warp: true only when no lane gave up
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* failed) {
    return __all_sync(0xffffffffu, mbar_wait_or_fail(bar, parity, failed));
}

// tf32_split without its branch on Inf and NaN: there lo = x - hi is NaN (a NaN's hi may be any value), which shows
// in the residual just as well; the converting warps are bound by their instructions.
__device__ __forceinline__ float tf32_hi(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}
// split four consecutive k of a row and store them at `addr` (hi) and `addr + part` (lo)
__device__ __forceinline__ void split_store4(uint32_t addr, uint32_t part, float4 x) {
    const float h0 = tf32_hi(x.x), h1 = tf32_hi(x.y), h2 = tf32_hi(x.z), h3 = tf32_hi(x.w);
    st_shared4(addr, h0, h1, h2, h3);
    st_shared4(addr + part, x.x - h0, x.y - h1, x.z - h2, x.w - h3);
}
// 8 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void umma_tf32_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the products of a 32-wide k panel: four k steps of lo.hi + hi.lo + hi.hi
__device__ __forceinline__ void umma_panel(uint32_t d, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi, uint32_t b_lo,
                                           uint32_t idesc, bool begin) {
    const uint64_t ah = umma_desc(a_hi, kKmajorLBO, kKmajorSBO), al = umma_desc(a_lo, kKmajorLBO, kKmajorSBO);
    const uint64_t bh = umma_desc(b_hi, kKmajorLBO, kKmajorSBO), bl = umma_desc(b_lo, kKmajorLBO, kKmajorSBO);
#pragma unroll
    for (int ks = 0; ks < kTcKC / 8; ks++) {           // 8 k are two core matrices, 256 bytes: 16 descriptor units
        umma_tf32_ss(d, al + 16 * ks, bh + 16 * ks, idesc, begin && ks == 0 ? 0u : 1u);
        umma_tf32_ss(d, ah + 16 * ks, bl + 16 * ks, idesc, 1u);
        umma_tf32_ss(d, ah + 16 * ks, bh + 16 * ks, idesc, 1u);
    }
}

// ITEMS: column pairs of a field panel per thread (n / 128 rounded up for the planes, 1 for z); AHEAD: panels in
// registers before they are stored.
template <int MODE, int ITEMS, int AHEAD>
__device__ void tc_pair_body(const TcPairArgs& g, const Blk& blk, bool first) {
    constexpr bool Z_MODE = MODE == kTcPairZ, F64 = MODE == kTcPairForward;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[kTcPairMaxStages], empty[kTcPairMaxStages], done[3];
    __shared__ uint32_t tmem_base;
    __shared__ int failed_flag;
    volatile int* failed = &failed_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int plane = nx * ny;
    const int m0 = blk.x * kTcRows, z = blk.y;                            // m0: first row y' (planes) or column n (z)
    const int N = g.n, NS = g.stages, tiles = g.tiles;
    const int k1 = Z_MODE ? nz : ny;                                      // the first product's K
    const int p1 = (k1 + kTcKC - 1) / kTcKC, p2 = N / kTcKC;              // panels of the two products
    const int n2 = Z_MODE ? N : min(kTcRows, (ny - m0 + 15) / 16 * 16);   // columns of the second product
    // a stage: slot 0 holds a 128-row operand (the first product's A, the second's converted one), slot 1 the other;
    // each as hi then lo parts
    const uint32_t stage_bytes = 2 * kTcPairPartA + g.slot1;
    const uint32_t part1 = N * kTcKC * 4, part2 = Z_MODE ? part1 : (uint32_t)tiles * kTcPairPartA;   // slot 1's parts
    const uint32_t sbase = smem_addr(smem);
    uint32_t cols = 32;
    while (cols < (uint32_t)(N + (Z_MODE ? N : tiles * kTcRows))) cols *= 2;

    // the basis panel of ring position `it` into its stage (one thread)
    auto copy_basis = [&](int it) {
        const int s = it % NS;
        uint64_t* bar = &full[s];
        const bool one = it < p1, slot0 = one && !Z_MODE;
        const uint32_t dst = sbase + s * stage_bytes + (slot0 ? 0 : 2 * kTcPairPartA);
        const uint32_t part = slot0 ? kTcPairPartA : one ? part1 : part2;
        const long long src = (one ? (long long)it * g.r1 + (slot0 ? m0 : 0) : (long long)(it - p1) * g.r2) * kTcKC;
        mbar_expect_tx(bar, 2 * part);
        for (int i = 0; i < 2; i++) bulk_copy(dst + i * part, (one ? g.basis1[i] : g.basis2[i]) + src, part, bar);
    };

    pdl_launch_dependents();
    if (warp == kTcPairConv / 32) tmem_alloc(&tmem_base, cols);
    if (tid == kTcPairConv + 32) {
        for (int s = 0; s < kTcPairMaxStages; s++) {
            mbar_init(&full[s], kTcPairConv / 32 + 1);       // the converting warps and the basis copy
            mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < 3; i++) mbar_init(&done[i], 1);
        failed_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        fence_async_smem();
        for (int it = 0; it < NS && it < p1 + p2; it++) copy_basis(it);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    pdl_wait();
    if (g.clear_condition && tid == 0 && first) cudaGraphSetConditional(g.handle, 0u);
    const Control* c = g.c;
    const bool converts = warp < kTcPairConv / 32;
    // the field's panels in registers: a thread takes 4 consecutive k (rows of the field) of the column pairs r_t + 128 j,
    // so that a warp reads 32 consecutive pairs.  Where the control block does not choose the field its first loads go
    // out before the block is read.
    using E2 = std::conditional_t<F64, double2, float2>;
    const int r_t = 2 * lane + 64 * (warp >> 3), k_t = 4 * (warp & 7);
    const int ld = Z_MODE ? plane : nx;
    const int width = Z_MODE ? plane - m0 : nx;                           // columns of the field, rows of its operand
    E2 buf[AHEAD][ITEMS][4];
    auto load = [&](E2 (&f)[ITEMS][4], const auto* F, int p) {
        const int k = p * kTcKC + k_t;
        const auto* q = F + (long long)k * ld;
#pragma unroll
        for (int i = 0; i < 4; i++, q += ld)
#pragma unroll
            for (int j = 0; j < ITEMS; j++)
                f[j][i] = k + i < k1 && r_t + 128 * j < width ? __ldg(reinterpret_cast<const E2*>(q + 128 * j)) : E2{0, 0};
    };
    const float* in = F64 ? nullptr : g.in + (Z_MODE ? (long long)m0 : (long long)z * plane) + r_t;
    if constexpr (!F64)
        if (converts) {
#pragma unroll
            for (int i = 0; i < AHEAD; i++)
                if (i < p1) load(buf[i], in, i);
        }
    const int err = c->error, use_rhs = c->use_rhs, reset = c->reset_phi, cond = c->cond;
    const double rhs2 = c->rhs_norm2, res2 = c->res_norm2;
    const double r2 = use_rhs ? rhs2 : res2;
    const bool live = !err && cond && r2 > 0;          // else no pass (backend.cu:803-804)

    if (warp == kTcPairConv / 32 + 1) {
        if (lane == 0) {
            int issued = min(NS, p1 + p2);
            for (; live && issued < p1 + p2; issued++) {
                if (!mbar_wait_or_fail(&empty[issued % NS], (issued / NS - 1) & 1, failed)) break;
                copy_basis(issued);
            }
            // a block with nothing to do, or that failed, stays until the copies have landed: it stands in for the
            // converting warps
            if (!live || *failed)
                for (int it = max(0, issued - NS); it < issued; it++) {
                    for (int w = 0; w < kTcPairConv / 32 && !live; w++) mbar_arrive(&full[it % NS]);
                    mbar_wait_bounded(&full[it % NS], (it / NS) & 1);
                }
        }
    } else if (warp == kTcPairConv / 32) {
        const uint32_t idesc1 = umma_idesc_tf32(kTcRows, N, 0, 0), idesc2 = umma_idesc_tf32(kTcRows, n2, 0, 0);
        if (lane == 0 && live) {
            bool ok = true;
            for (int it = 0; it < p1 + p2; it++) {
                const int s = it % NS;
                if (!(ok = mbar_wait_or_fail(&full[s], (it / NS) & 1, failed))) break;
                if (it == p1) tc_fence_after();
                const uint32_t s0 = sbase + s * stage_bytes, s1 = s0 + 2 * kTcPairPartA;
                if (it < p1) {
                    umma_panel(tmem, s0, s0 + kTcPairPartA, s1, s1 + part1, idesc1, it == 0);
                } else if (Z_MODE) {
                    umma_panel(tmem + N, s0, s0 + kTcPairPartA, s1, s1 + part1, idesc1, it == p1);
                } else {
                    for (int m = 0; m < tiles; m++)
                        umma_panel(tmem + N + m * kTcRows, s1 + m * kTcPairPartA, s1 + part2 + m * kTcPairPartA, s0,
                                   s0 + kTcPairPartA, idesc2, it == p1);
                }
                umma_commit(&empty[s]);
                if (it == p1 - 1) umma_commit(&done[0]);
                if (it == p1 + p2 - 1) umma_commit(&done[1]);
            }
            if (!ok) {                          // the MMAs already issued end before the block leaves
                umma_commit(&done[2]);
                mbar_wait_bounded(&done[2], 0);
            }
        }
    } else if (live) {
        const double rms = Z_MODE ? 1.0 : sqrt(r2 / g.n_cell);
        bool ok = true;
        // the other operand of what follows the products comes into L2 meanwhile: 1/lambda's columns, phi's rows
        if constexpr (Z_MODE) {
            for (int i = tid; i < nz * 4; i += kTcPairConv)
                if (m0 + (i & 3) * 32 < plane) prefetch_l2(g.inv_lambda + (long long)(i >> 2) * plane + m0 + (i & 3) * 32);
        } else if constexpr (!F64) {
            const int count = min(kTcRows, ny - m0) * nx;
            const double* q = g.phi + (long long)z * plane + m0 * nx;
            for (int i = tid * 16; i < count && !reset; i += kTcPairConv * 16) prefetch_l2(q + i);
        }
        auto publish = [&](int it) {
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[it % NS]);
        };
        // ---- first product.  The two rows of a pair go out in the order that gives the 8 lanes of a quarter warp 8
        // different rows of their core matrices (no bank conflicts).
        {
            const double inv_rms = 1.0 / rms;
            const int rows = Z_MODE ? kTcRows : N, swap = (lane >> 2) & 1;
            const uint32_t dst0 = sbase + (Z_MODE ? 0 : 2 * kTcPairPartA) + kmajor_off(r_t, k_t);
            const uint32_t part = Z_MODE ? (uint32_t)kTcPairPartA : part1;
            const double* r = nullptr;
            if constexpr (F64) {
                r = (use_rhs && g.r_alt ? g.r_alt : g.r) + (long long)z * plane + r_t;
#pragma unroll
                for (int i = 0; i < AHEAD; i++)
                    if (i < p1) load(buf[i], r, i);
            }
#pragma unroll 1
            for (int p0 = 0; ok && p0 < p1; p0 += AHEAD) {
#pragma unroll
                for (int i = 0; i < AHEAD; i++) {
                    const int p = p0 + i;
                    if (!ok || p >= p1) break;
                    const int s = p % NS;
                    if (p >= NS && !mbar_wait_warp(&empty[s], (p / NS - 1) & 1, failed)) { ok = false; break; }
                    const uint32_t dst = dst0 + s * stage_bytes;
#pragma unroll
                    for (int j = 0; j < ITEMS; j++) {
                        if (r_t + 128 * j >= rows) break;
                        float4 a, b;
                        const E2* v = buf[i][j];
                        if constexpr (F64) {
                            a = make_float4((float)(v[0].x * inv_rms), (float)(v[1].x * inv_rms), (float)(v[2].x * inv_rms),
                                            (float)(v[3].x * inv_rms));
                            b = make_float4((float)(v[0].y * inv_rms), (float)(v[1].y * inv_rms), (float)(v[2].y * inv_rms),
                                            (float)(v[3].y * inv_rms));
                        } else {
                            a = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
                            b = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
                        }
                        const uint32_t at = dst + j * 16384;
                        split_store4(at + 16 * swap, part, swap ? b : a);
                        split_store4(at + 16 - 16 * swap, part, swap ? a : b);
                    }
                    publish(p);
                    if (p + AHEAD < p1) {
                        if constexpr (F64) load(buf[i], r, p + AHEAD);
                        else load(buf[i], in, p + AHEAD);
                    }
                }
            }
        }
        // ---- second product: the first result out of TMEM (times 1/lambda for z), this warp's 32 lanes and 8 of the
        // panel's 32 columns
        const int lb = warp & 3, quarter = warp >> 2, row = lb * 32 + lane;
        const uint32_t tlane = tmem + ((uint32_t)(lb * 32) << 16);
        if (ok) {
            float il[2][8];
            auto load_lambda = [&](float (&l)[8], int p) {
                if constexpr (Z_MODE) {
                    const int zz = p * kTcKC + 8 * quarter;
                    const float* q = g.inv_lambda + (long long)zz * plane + m0 + row;
#pragma unroll
                    for (int j = 0; j < 8; j++, q += plane) l[j] = m0 + row < plane && zz + j < nz ? __ldg(q) : 0.f;
                }
            };
            load_lambda(il[0], 0);
            load_lambda(il[1], 1);
            ok = mbar_wait_warp(&done[0], 0, failed);
            tc_fence_after();
            auto convert = [&](float (&l)[8], int p) {
                const int it = p1 + p, s = it % NS;
                float v[8];
                __syncwarp();
                tmem_ld8(tlane + p * kTcKC + 8 * quarter, v);
                if constexpr (Z_MODE) {
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] *= l[j];
                    load_lambda(l, p + 2);
                }
                if (it >= NS && !mbar_wait_warp(&empty[s], (it / NS - 1) & 1, failed)) { ok = false; return; }
                const uint32_t dst = sbase + s * stage_bytes + kmajor_off(row, 8 * quarter);
                split_store4(dst, kTcPairPartA, make_float4(v[0], v[1], v[2], v[3]));
                split_store4(dst + 128, kTcPairPartA, make_float4(v[4], v[5], v[6], v[7]));
                publish(it);
            };
#pragma unroll 1
            for (int p = 0; ok && p < p2; p += 2) {
                convert(il[0], p);
                if (ok && p + 1 < p2) convert(il[1], p + 1);
            }
        }
        // ---- the outcome: this warp's 32 lanes, every fourth group of 8 columns
        const int count = Z_MODE ? nz : min(kTcRows, ny - m0);                 // columns that exist
        const int width = Z_MODE ? plane - m0 : nx;                            // rows (lanes) that exist
        const int step = Z_MODE ? plane : nx;
        const long long base = Z_MODE ? (long long)m0 : (long long)z * plane + (long long)m0 * nx;
        constexpr bool ADD = MODE == kTcPairInverse;
        double old[2][8];
        auto load_phi = [&](double (&o)[8], int m, int c0) {
            if constexpr (ADD) {
                const int x = m * kTcRows + row;
                const double* q = g.phi + base + (long long)c0 * step + x;
#pragma unroll
                for (int j = 0; j < 8; j++, q += step) o[j] = x < width && c0 + j < count && !reset ? *q : 0.0;
            }
        };
        load_phi(old[0], 0, 8 * quarter);
        if (ok) ok = mbar_wait_warp(&done[1], 0, failed);
        tc_fence_after();
        for (int m = 0; ok && m < tiles; m++) {
            const int x = m * kTcRows + row;
            auto put = [&](double (&o)[8], double (&next)[8], int c0) {
                float v[8];
                __syncwarp();
                tmem_ld8(tlane + N + m * kTcRows + c0, v);
                if (c0 + 32 < count) load_phi(next, m, c0 + 32);
                else if (m + 1 < tiles) load_phi(next, m + 1, 8 * quarter);
                if (x >= width) return;
                if constexpr (ADD) {
                    double* q = g.phi + base + (long long)c0 * step + x;
#pragma unroll
                    for (int j = 0; j < 8; j++, q += step)
                        if (c0 + j < count) *q = o[j] + (double)v[j] * rms;
                } else {
                    float* q = g.out + base + (long long)c0 * step + x;
#pragma unroll
                    for (int j = 0; j < 8; j++, q += step)
                        if (c0 + j < count) *q = v[j];
                }
            };
#pragma unroll 1
            for (int c0 = 8 * quarter; c0 < count; c0 += 64) {
                put(old[0], old[1], c0);
                if (c0 + 32 < count) {
                    put(old[1], old[0], c0 + 32);
                } else if constexpr (ADD) {
#pragma unroll
                    for (int j = 0; j < 8; j++) old[0][j] = old[1][j];         // the next tile's first group
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (failed_flag && tid == 0) atomicExch(g.error, (int)kDeviceWait);
    if (warp == kTcPairConv / 32) tmem_dealloc(tmem, cols);
}

template <int MODE, int ITEMS> struct TcPairAhead {
    // panels of values held in registers until they are stored: at most 64 registers
    static constexpr int value = MODE == kTcPairForward ? (ITEMS > 1 ? 2 : 3) : (ITEMS > 1 ? 3 : 4);
};
template <int MODE, int ITEMS>
__global__ void __launch_bounds__(kTcPairThreads, 1) tc_pair_kernel(TcPairArgs g) {
    tc_pair_body<MODE, ITEMS, TcPairAhead<MODE, ITEMS>::value>(g, real_blk(), first_block());
}
// a batch of cavities: grid x runs over the work list (BatchItem)
template <int MODE, int ITEMS>
__global__ void __launch_bounds__(kTcPairThreads, 1) tc_pair_batched(const TcPairArgs* args, const BatchItem* items,
                                                                     const int* live) {
    __shared__ TcPairArgs g;
    int cav;
    const Blk k = item_blk(items, live, cav);
    if (cav < 0) {
        if (MODE == kTcPairForward) dead_slot_clear(args, items);
        return;
    }
    load_args(g, args + cav);
    tc_pair_body<MODE, ITEMS, TcPairAhead<MODE, ITEMS>::value>(g, k, first_block());
}

// ---------------------------------------------------------------- host side
constexpr size_t kTcPairSmemMax = 224 * 1024;      // of the 227 KB a block may have, less the static part
constexpr size_t kTcPairSmemMin = 120 * 1024;      // one CTA per SM: its TMEM columns (up to 512) are the SM's
struct TcPairShape {
    int n, tiles, slot1, stages, items;
    size_t smem;
};
inline bool tc_pair_fits(int nx, int ny, int nz) {
    return nx % 4 == 0 && nx <= kTcPairMax && ny <= kTcPairMax && nz <= kTcPairMax;
}
// Whether a pass runs as paired launches: wherever the axes allow, unless CAVITY_TC_KERNEL names one of the six-launch
// kernels; in a batch as the batch decides for all its members.
inline bool tc_pair_used(int nx, int ny, int nz) {
    if (tc_kernel_forced() >= 0) return false;
    if (g_launch_record) return g_batch_tc_pairs > 0;
    return tc_pair_fits(nx, ny, nz);
}
inline TcPairShape tc_pair_shape(int mode, int nx, int ny, int nz) {
    const bool z = mode == kTcPairZ;
    TcPairShape s;
    s.n = ((z ? nz : nx) + 31) / 32 * 32;
    s.tiles = z ? 1 : (nx + kTcRows - 1) / kTcRows;
    s.slot1 = std::max(2 * s.n * kTcKC * 4, z ? 0 : 2 * s.tiles * kTcPairPartA);
    const size_t stage = 2 * (size_t)kTcPairPartA + s.slot1;
    const int panels = ((z ? nz : ny) + kTcKC - 1) / kTcKC + s.n / kTcKC;
    s.stages = (int)std::min<size_t>(std::min<size_t>(kTcPairMaxStages, kTcPairSmemMax / stage), (size_t)panels);
    s.items = z || s.n <= 128 ? 1 : 2;
    s.smem = std::max(kTcPairSmemMin, s.stages * stage);
    if (g_launch_record && g_batch_tc_pairs == 2) {      // members of several sizes share one variant of the kernel
        s.items = z ? 1 : 2;
        s.smem = kTcPairSmemMax;
    }
    return s;
}
inline dim3 tc_pair_grid(int mode, int nx, int ny, int nz) {
    if (mode == kTcPairZ) return dim3((unsigned int)(((long long)nx * ny + kTcRows - 1) / kTcRows));
    return dim3((ny + kTcRows - 1) / kTcRows, nz);
}
// variant code of a recorded launch: mode, items
inline int tc_pair_variant(int mode, int items) { return mode | (items << 4); }

template <class F> inline void tc_pair_dispatch(int mode, int items, F&& f) {
    using std::integral_constant;
    if (mode == kTcPairZ) f(integral_constant<int, kTcPairZ>{}, integral_constant<int, 1>{});
    else if (mode == kTcPairForward && items == 1) f(integral_constant<int, kTcPairForward>{}, integral_constant<int, 1>{});
    else if (mode == kTcPairForward) f(integral_constant<int, kTcPairForward>{}, integral_constant<int, 2>{});
    else if (items == 1) f(integral_constant<int, kTcPairInverse>{}, integral_constant<int, 1>{});
    else f(integral_constant<int, kTcPairInverse>{}, integral_constant<int, 2>{});
}
// once per process, before any capture: the dynamic shared memory of every instance
inline cudaError_t tc_pair_prepare() {
    static const cudaError_t e = [] {
        cudaError_t r = cudaSuccess;
        for (int mode = 0; mode < 3; mode++)
            for (int items = 1; items <= 2; items++)
                tc_pair_dispatch(mode, items, [&](auto m, auto i) {
                    if (r == cudaSuccess)
                        r = cudaFuncSetAttribute(tc_pair_kernel<m(), i()>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kTcPairSmemMax);
                    if (r == cudaSuccess)
                        r = cudaFuncSetAttribute(tc_pair_batched<m(), i()>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kTcPairSmemMax);
                });
        return r;
    }();
    return e;
}
inline void launch_tc_pair_batched(int variant, dim3 grid, size_t smem, const BatchItem* items, const int* live,
                                   const TcPairArgs* d, cudaStream_t st) {
    tc_pair_dispatch(variant & 15, variant >> 4, [&](auto m, auto i) {
        launch_pdl(tc_pair_batched<m(), i()>, grid, dim3(kTcPairThreads), smem, st, d, items, live);
    });
}

// One pass as three launches (arguments as launch_tc_fdm_pass)
inline void launch_tc_fdm_pass_pairs(cudaStream_t st, const TcFdmOperands& op, const double* r, const double* r_alt,
                                     double* phi, float* t1, float* t2, Control* c, cudaGraphConditionalHandle h, bool clear) {
    const int n[3] = {op.nx, op.ny, op.nz};
    for (int mode = 0; mode < 3; mode++) {
        const TcPairShape s = tc_pair_shape(mode, op.nx, op.ny, op.nz);
        TcPairArgs g = {};
        g.nx = op.nx; g.ny = op.ny; g.nz = op.nz;
        g.n = s.n; g.tiles = s.tiles; g.slot1 = s.slot1; g.stages = s.stages;
        // the axes of the two products, and S^T (images 2, 3: rows are the transformed index) or S (0, 1) of each
        const int a1 = mode == kTcPairZ ? 2 : 1, a2 = mode == kTcPairZ ? 2 : 0;
        const int i1 = mode == kTcPairInverse ? 0 : 2, i2 = mode == kTcPairForward ? 2 : 0;
        g.basis1[0] = op.img[a1][i1]; g.basis1[1] = op.img[a1][i1 + 1]; g.r1 = basis_image_rows(n[a1]);
        g.basis2[0] = op.img[a2][i2]; g.basis2[1] = op.img[a2][i2 + 1]; g.r2 = basis_image_rows(n[a2]);
        g.r = r; g.r_alt = r_alt;
        g.in = mode == kTcPairZ ? t1 : t2;
        g.out = mode == kTcPairForward ? t1 : t2;
        g.inv_lambda = op.inv_lambda;
        g.phi = phi;
        g.n_cell = (double)op.nx * op.ny * op.nz;
        g.c = c;
        g.error = &c->error;
        g.handle = h;
        g.clear_condition = clear && mode == kTcPairForward;
        const dim3 grid = tc_pair_grid(mode, op.nx, op.ny, op.nz);
        if (record_launch(kLkTcPair, tc_pair_variant(mode, s.items), grid, s.smem, g)) continue;
        tc_pair_dispatch(mode, s.items, [&](auto m, auto i) {
            launch_pdl(tc_pair_kernel<m(), i()>, grid, dim3(kTcPairThreads), s.smem, st, g);
        });
    }
}

// One pass of the mixed form (arguments as launch_tc_fdm_pass): three paired launches, or six single transforms
inline void launch_tc_pass(cudaStream_t st, const TcFdmOperands& op, const double* r, const double* r_alt, double* phi,
                           float* t1, float* t2, Control* c, cudaGraphConditionalHandle h, bool clear, int sms) {
    if (tc_pair_used(op.nx, op.ny, op.nz)) launch_tc_fdm_pass_pairs(st, op, r, r_alt, phi, t1, t2, c, h, clear);
    else launch_tc_fdm_pass(st, op, r, r_alt, phi, t1, t2, c, h, clear, sms);
}

}  // namespace cavity
