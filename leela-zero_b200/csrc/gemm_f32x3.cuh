// The 36 channel contractions in fp32, on the tensor cores:
//   M[t][p][k] = sum_c V[t][p][c] * U[t][k][c],   t = 0..35
// Every operand is carried as three bf16 planes, x = x0 + x1 + x2 with x0 =
// bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1): three 8-bit significands
// hold the 24 bits of an fp32 number, so the split loses nothing.  Of the nine
// products of planes the six down to 2^-16 are summed (x0y0, x0y1, x1y0, x1y1,
// x0y2, x2y0); what is left out is below 2^-26 of the product, an eighth of the
// rounding an fp32 product itself would have.
//
// Accumulation.  The tensor core adds to an fp32 accumulator but truncates, so
// what counts is how often a large sum is added to.  The five small products
// (2^-8 and below) therefore have an accumulator of their own, whose truncations
// are 2^-8 of the sum's last place, and x0y0 has two, one for each half of the
// reduction; the epilogue adds the three in fp32.  Measured against fp64 (128 x 128
// outputs, normal operands), relative error of the result: reduction length 64 /
// 128 / 256 / 512: 7.2e-8 / 7.3e-8 / 1.2e-7 / 2.3e-7, where a chain of fp32 FMAs
// has 1.5e-7 / 2.0e-7 / 2.9e-7 / 4.1e-7; with all six products in one accumulator
// it is 1.4e-6 at 256.
//
// V is [36 * Pa rows][3 * Cin] and U [36 * Kp rows][3 * Cin], plane-major within a
// row.  One work item is (t, slice of N output channels, block of 128 rows);
// items are numbered row block innermost, so that neighbouring CTAs share U in L2.
// A pipeline stage is one 64-channel chunk: three V tiles and three U tiles, each
// plane pair with a "full" barrier of its own, because x0y0 can start while the
// other planes are on their way.  N = 128 normally, 64 where that gives the SMs
// more items than N = 128 has (small batches).
//
// Roles as in gemm_tcgen05.cuh with eight epilogue warps.  The small accumulator
// alternates between two places; the two x0y0 ones are free again as soon as the
// epilogue has read them, which it does first.
//
// What bounds it: at 256 x 256 channels the MMAs (96 of 128 x 128 x 16 per item at
// 65 cycles) against 96 KB of operands per 24 of them, 61 bytes a cycle and SM.
#pragma once
#include "gemm_tcgen05.cuh"

namespace lzb {
namespace f3 {

using namespace tc;

constexpr int kF3Threads = 320;                        // producer, MMA, 8 epilogue warps
constexpr uint32_t kATile = kBlockM * 128;             // 16 KB: one plane of 128 rows x 64 channels
template <int N> struct Shape {
    static constexpr uint32_t b_tile = N * 128;
    static constexpr uint32_t stage = 3 * (kATile + b_tile);
    static constexpr int stages = N == 64 ? 3 : 2;
    static constexpr uint32_t smem = stages * stage + kBarBytes + 1024;
};
static_assert(Shape<64>::smem <= 227 * 1024 && Shape<128>::smem <= 227 * 1024, "shared memory of one CTA");

constexpr int kErrF3Producer = 601;
constexpr int kErrF3Mma = 602;
constexpr int kErrF3Epilogue = 603;

// Split an fp32 value into its three bf16 planes.
__device__ __forceinline__ void split3(float v, __nv_bfloat16& p0, __nv_bfloat16& p1, __nv_bfloat16& p2) {
    p0 = __float2bfloat16_rn(v);
    const float r1 = v - __bfloat162float(p0);           // exact
    p1 = __float2bfloat16_rn(r1);
    p2 = __float2bfloat16_rn(r1 - __bfloat162float(p1));
}

// tmV : [36 * Pa][3 * Cin], box 64 x 128; tmV32 : the same, box 64 x 32 (the last
// rows of a small batch); tmU : [36 * Kp][3 * Cin], box 64 x N.  nblk row blocks of
// 128 covering P rows.
template <int N>
__global__ void __launch_bounds__(kF3Threads, 1) gemm_f32x3_kernel(
    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmV32,
    const __grid_constant__ CUtensorMap tmU, float* M, int Pa, int P, int Kp, int Cin, int nblk, int* err) {
    using S = Shape<N>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (base - raw);
    unsigned char* bar_mem = smem + S::stages * S::stage;
    const uint32_t bars = smem_u32(bar_mem);
    auto full_bar = [&](int s, int plane) { return bars + 8u * (s * 3 + plane); };
    auto empty_bar = [&](int s) { return bars + 8u * (12 + s); };
    auto tfull_bar = [&](int a) { return bars + 8u * (16 + a); };       // all accumulators of an item
    auto sfree_bar = [&](int a) { return bars + 8u * (18 + a); };       // small accumulator a
    const uint32_t mfree_bar = bars + 8u * 20;                           // both x0y0 accumulators
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_mem + 8 * 24);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_mem + 8 * 24 + 8);

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S::stages; s++) {
            for (int k = 0; k < 3; k++) mbar_init(full_bar(s, k), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(sfree_bar(a), 8);
        }
        mbar_init(mfree_bar, 8);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t*>(tmem_slot))),
                     "r"(4u * N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // columns: [x0y0 first half][x0y0 second half][small 0][small 1], N each
    const int chunks = Cin / kChunkK, first_half = (chunks + 1) / 2;
    const int slices = Kp / N, items = kPoints * slices * nblk;
    const int item_begin = static_cast<int>(static_cast<long long>(blockIdx.x) * items / gridDim.x);
    const int item_end = static_cast<int>(static_cast<long long>(blockIdx.x + 1) * items / gridDim.x);

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true, waited = false;
            // U does not depend on the previous kernel: the first stages' tiles are
            // requested before this kernel waits for V
            const int ahead = item_begin < item_end ? (chunks < S::stages ? chunks : S::stages) : 0;
            auto load_u = [&](int item, int c, int s) {
                const int ts = item / nblk;                    // t * slices + slice
                const int row = (ts / slices) * Kp + (ts % slices) * N;
                for (int k = 0; k < 3; k++) {
                    tma_load_2d(base + s * S::stage + 3 * kATile + k * S::b_tile, &tmU, k * Cin + c * kChunkK, row,
                                full_bar(s, k));
                }
            };
            auto expect = [&](int item, int s) {
                const int left = P - (item % nblk) * kBlockM;
                const uint32_t a = left >= kBlockM ? kATile : static_cast<uint32_t>((left + 31) / 32) * 32u * 128u;
                for (int k = 0; k < 3; k++) mbar_expect_tx(full_bar(s, k), a + S::b_tile);
            };
            for (int c = 0; c < ahead; ++c) {
                expect(item_begin, c);
                load_u(item_begin, c, c);
            }
            for (int item = item_begin; item < item_end && ok; ++item) {
                const int t = item / nblk / slices, blk = item % nblk;
                const int left = P - blk * kBlockM, row = t * Pa + blk * kBlockM;
                for (int c = 0; c < chunks; ++c) {
                    if (item != item_begin || c >= ahead) {
                        ok = mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, err, kErrF3Producer);
                        if (!ok) break;
                        expect(item, stage);
                        load_u(item, c, stage);
                    }
                    if (!waited) {
                        asm volatile("griddepcontrol.wait;" ::: "memory");
                        waited = true;
                    }
                    for (int k = 0; k < 3; k++) {
                        const uint32_t dst = base + stage * S::stage + k * kATile;
                        if (left >= kBlockM) {
                            tma_load_2d(dst, &tmV, k * Cin + c * kChunkK, row, full_bar(stage, k));
                        } else {
                            for (int r = 0; r < left; r += 32) {
                                tma_load_2d(dst + r * 128, &tmV32, k * Cin + c * kChunkK, row + r,
                                            full_bar(stage, k));
                            }
                        }
                    }
                    if (++stage == S::stages) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
                                   (static_cast<uint32_t>(kBlockM >> 4) << 24);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int local = 0;
            const uint64_t d0 = umma_desc_sw128(base);
            for (int item = item_begin; item < item_end && ok; ++item, ++local) {
                const int acc = local & 1;
                const uint32_t t_small = tmem_base + static_cast<uint32_t>((2 + acc) * N);
                ok = mbar_wait(sfree_bar(acc), ((local >> 1) & 1u) ^ 1u, abort_flag, err, kErrF3Mma);
                for (int c = 0; c < chunks && ok; ++c) {
                    const uint32_t t_main = tmem_base + (c < first_half ? 0u : static_cast<uint32_t>(N));
                    const uint64_t s16 = static_cast<uint64_t>(stage) * (S::stage >> 4);
                    auto a = [&](int k) { return d0 + s16 + static_cast<uint64_t>(k) * (kATile >> 4); };
                    auto b = [&](int k) {
                        return d0 + s16 + (3 * kATile >> 4) + static_cast<uint64_t>(k) * (S::b_tile >> 4);
                    };
                    if (c == 0) ok = mbar_wait(mfree_bar, (local & 1u) ^ 1u, abort_flag, err, kErrF3Mma);
                    if (ok) ok = mbar_wait(full_bar(stage, 0), phase, abort_flag, err, kErrF3Mma);
                    if (!ok) break;
                    tcgen05_fence_after();
                    if (c == 0 || c == first_half) tcgen05_mma_f16<false>(t_main, a(0), b(0), idesc);
                    else tcgen05_mma_f16<true>(t_main, a(0), b(0), idesc);
#pragma unroll
                    for (int k = 1; k < 4; ++k) tcgen05_mma_f16<true>(t_main, a(0) + 2u * k, b(0) + 2u * k, idesc);
                    ok = mbar_wait(full_bar(stage, 1), phase, abort_flag, err, kErrF3Mma);
                    if (!ok) break;
                    if (c == 0) tcgen05_mma_f16<false>(t_small, a(1), b(1), idesc);
                    else tcgen05_mma_f16<true>(t_small, a(1), b(1), idesc);
#pragma unroll
                    for (int k = 1; k < 4; ++k) tcgen05_mma_f16<true>(t_small, a(1) + 2u * k, b(1) + 2u * k, idesc);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tcgen05_mma_f16<true>(t_small, a(0) + 2u * k, b(1) + 2u * k, idesc);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tcgen05_mma_f16<true>(t_small, a(1) + 2u * k, b(0) + 2u * k, idesc);
                    ok = mbar_wait(full_bar(stage, 2), phase, abort_flag, err, kErrF3Mma);
                    if (!ok) break;
#pragma unroll
                    for (int k = 0; k < 4; ++k) tcgen05_mma_f16<true>(t_small, a(0) + 2u * k, b(2) + 2u * k, idesc);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tcgen05_mma_f16<true>(t_small, a(2) + 2u * k, b(0) + 2u * k, idesc);
                    tcgen05_commit(empty_bar(stage));
                    if (++stage == S::stages) { stage = 0; phase ^= 1u; }
                }
                tcgen05_commit(tfull_bar(acc));
            }
        }
    } else {
        // ------------------------------------------------ epilogue (warps 2..9)
        const int qd = warp & 3;
        constexpr int kCols = N / 2;                   // channels of this warp
        const int col0 = ((warp - 2) >> 2) * kCols;
        const uint32_t lanes = static_cast<uint32_t>(qd * 32) << 16;
        bool waited = false;
        int local = 0;
        for (int item = item_begin; item < item_end; ++item, ++local) {
            const int acc = local & 1;
            const int ts = item / nblk, t = ts / slices;
            const int p = (item % nblk) * kBlockM + qd * 32 + lane;
            bool ok = true;
            if (lane == 0) ok = mbar_wait(tfull_bar(acc), (local >> 1) & 1u, abort_flag, err, kErrF3Epilogue);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            tcgen05_fence_after();
            float sum[kCols];
#pragma unroll
            for (int j = 0; j < kCols; j += 32) {
                uint32_t r0[32];
                LZB_TMEM_LD32(r0, tmem_base + lanes + static_cast<uint32_t>(col0 + j));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 32; ++i) sum[j + i] = __uint_as_float(r0[i]);
                if (chunks > 1) {
                    LZB_TMEM_LD32(r0, tmem_base + lanes + static_cast<uint32_t>(N + col0 + j));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; ++i) sum[j + i] += __uint_as_float(r0[i]);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(mfree_bar);
#pragma unroll
            for (int j = 0; j < kCols; j += 32) {
                uint32_t r0[32];
                LZB_TMEM_LD32(r0, tmem_base + lanes + static_cast<uint32_t>((2 + acc) * N + col0 + j));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 32; ++i) sum[j + i] += __uint_as_float(r0[i]);
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(sfree_bar(acc));
            if (!waited) {
                // M may still be read by the kernel before this one
                asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
            }
            if (p < P) {
                float* dst = M + (static_cast<size_t>(t) * Pa + p) * Kp + (ts % slices) * N + col0;
                // whole 32-byte sectors per lane and store
#pragma unroll
                for (int j = 0; j < kCols; j += 8) {
                    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + j),
                                 "f"(sum[j]), "f"(sum[j + 1]), "f"(sum[j + 2]), "f"(sum[j + 3]), "f"(sum[j + 4]),
                                 "f"(sum[j + 5]), "f"(sum[j + 6]), "f"(sum[j + 7])
                                 : "memory");
                }
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(4u * N)
                     : "memory");
    }
}

}  // namespace f3
}  // namespace lzb
