// The network heads, from the last activations to policy and winrate in one launch:
//   policy: 1x1 conv to 2 planes, batch-norm + ReLU -> FC 722 -> 362 -> softmax
//   value : 1x1 conv to 1 plane,  batch-norm + ReLU -> FC 361 -> 256 ReLU
//           -> FC 256 -> 1 -> (1 + tanh) / 2
// This is the arithmetic of the convolutions in CPUPipe::forward
// (src/CPUPipe.cpp:301-350) and of what Network::get_output_internal runs on the
// CPU for every evaluation (src/Network.cpp:833-851, innerproduct :609-637,
// softmax :693-712).
//
// One CLUSTER of eight CTAs per position (or per group of positions).  Each CTA
// owns 46 of the 361 cells in all three planes: it computes the 1x1 convolutions
// of its cells, which are then exactly its slice of the inputs of both fully
// connected layers, and sends the partial sums of their outputs to the shared
// memory of the CTA that finishes a head (policy: the first, value: the second),
// which adds them in slice order.
//
// What bounds it is latency.  A thread owns one (plane, output) pair, 46 weights;
// it has them in registers before it waits for the tower, so that after the tower
// only the activations (L2), two block barriers and one cluster barrier remain.
// As separate launches (1x1 convolutions, policy head, value head), with the weights
// fetched four at a time behind the activations, the heads of one position took
// 25 us; together with the copies that followed them they were a third of a small
// evaluation.  With more positions than clusters fit the GPU at once a cluster
// takes several at a time: it reads the 1.4 MB of weights once for all of them, and
// each of its CTAs finishes another position.
#pragma once
#include "conv_direct.cuh"
#include "winograd_math.cuh"

namespace lzb {

constexpr int kMoves = 362;
constexpr int kValueHidden = 256;
constexpr int kHeadCtas = 8;                                    // CTAs per cluster
constexpr int kHeadCells = (kSq + kHeadCtas - 1) / kHeadCtas;   // 46 cells per CTA
constexpr int kHeadThreads = 992;                               // 362 + 362 + 256 (plane, output) pairs
static_assert(kHeadThreads >= 2 * kMoves + kValueHidden && kHeadThreads % 32 == 0, "a thread per pair");

__device__ __forceinline__ float block_reduce(float v, float* scratch, bool is_max) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, v, off);
        v = is_max ? fmaxf(v, o) : v + o;
    }
    __syncthreads();               // scratch may still be read from a previous call
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float r = scratch[0];
    for (int i = 1; i < nw; i++) r = is_max ? fmaxf(r, scratch[i]) : r + scratch[i];
    return r;
}
__device__ __forceinline__ uint32_t head_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// store into the shared memory of CTA `rank` of the cluster, at the offset `local` has here
__device__ __forceinline__ void store_to_cta(float* local, uint32_t rank, float v) {
    uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(local)), remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}
__device__ __forceinline__ void head_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The three 1x1 convolutions of one cell by one warp: channels two per lane, 64
// apart, added up the lanes.  Activations are rows of ldx elements; lo_off > 0:
// two planes, the low one lo_off elements after the high one, stored as T or, with
// lo_e5m2, as one e5m2 byte per channel.  w: [3][Cp].
template <typename T>
__device__ __forceinline__ float3 head_conv_cell(const T* x, const float* __restrict__ w, int Cp, int lo_off,
                                                 int lo_e5m2, int lane) {
    using P2 = Pair<T>;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
    for (int c = 2 * lane; c < Cp; c += 64) {
        float2 v = P2::to_f2(*reinterpret_cast<const typename P2::type*>(x + c));
        if (lo_off > 0 && lo_e5m2) {
            const unsigned short two =
                *reinterpret_cast<const unsigned short*>(reinterpret_cast<const unsigned char*>(x + lo_off) + c);
            v.x += dc::e5m2_to_float(two);
            v.y += dc::e5m2_to_float(two >> 8);
        } else if (lo_off > 0) {
            const float2 l = P2::to_f2(*reinterpret_cast<const typename P2::type*>(x + lo_off + c));
            v.x += l.x;
            v.y += l.y;
        }
        const float2 w0 = *reinterpret_cast<const float2*>(w + c);
        const float2 w1 = *reinterpret_cast<const float2*>(w + Cp + c);
        const float2 w2 = *reinterpret_cast<const float2*>(w + 2 * Cp + c);
        a0 += w0.x * v.x + w0.y * v.y;
        a1 += w1.x * v.x + w1.y * v.y;
        a2 += w2.x * v.x + w2.y * v.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, off);
        a1 += __shfl_xor_sync(0xffffffffu, a1, off);
        a2 += __shfl_xor_sync(0xffffffffu, a2, off);
    }
    return make_float3(a0, a1, a2);
}
// Row of board cell s of position n: padded cell-major layout (conv_direct.cuh), or
// 361 dense rows per position (the Winograd pipeline).
template <bool kCells>
__device__ __forceinline__ size_t head_row(int n, int s) {
    if (kCells) return static_cast<size_t>(dc::cell_of(n, s / kBoard, s % kBoard));
    return static_cast<size_t>(n) * kSq + s;
}

// Raw head planes pol[n][2][361], val[n][361] (which may be page-locked host memory):
// 32 board cells per CTA, four per warp, written as whole rows of 128 bytes.
// err_out, if given, receives *err; run, if given, counts the tower run that ends here.
template <typename T, bool kCells>
__global__ void __launch_bounds__(256) head_planes_kernel(const T* X, const float* __restrict__ w, int Cp, int n,
                                                          float* __restrict__ pol, float* __restrict__ val, int ldx,
                                                          int lo_off, int lo_e5m2, const int* err, int* err_out,
                                                          uint32_t* run) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (err_out != nullptr) *err_out = *err;
        if (run != nullptr) *run += 1u;
    }
    __shared__ float out[3][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = blockIdx.x * 32;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int cell = first + warp * 4 + k;
        if (cell >= n * kSq) break;
        const float3 r = head_conv_cell<T>(X + head_row<kCells>(cell / kSq, cell % kSq) * ldx, w, Cp, lo_off,
                                           lo_e5m2, lane);
        if (lane == 0) {
            out[0][warp * 4 + k] = r.x;
            out[1][warp * 4 + k] = r.y;
            out[2][warp * 4 + k] = r.z;
        }
    }
    __syncthreads();
    const int cell = first + lane;
    if (warp < 3 && cell < n * kSq) {
        const int pos = cell / kSq, s = cell % kSq;
        if (warp < 2) pol[((size_t)pos * 2 + warp) * kSq + s] = out[warp][lane];
        else val[(size_t)pos * kSq + s] = out[2][lane];
    }
}

struct HeadWeights {
    const float *bn_pol_mean, *bn_pol_invstd, *ip_pol_wT /*[722][362]*/, *ip_pol_b, *bn_val_mean, *bn_val_invstd,
        *ip1_val_wT /*[361][256]*/, *ip1_val_b, *ip2_val_w, *ip2_val_b;
};

// grid: clusters of kHeadCtas.  A cluster takes its positions G = kHeadGroup at a
// time, first group at G * cluster, and CTA g of the cluster finishes position g of
// a group (its value head is finished by the next CTA, so that with one position
// the two heads end side by side).
template <typename T, bool kCells, int kHeadGroup>
__global__ void __cluster_dims__(kHeadCtas, 1, 1) __launch_bounds__(kHeadThreads)
    heads_kernel(const T* X, const float* __restrict__ w, int Cp, int n, int ldx, int lo_off, int lo_e5m2,
                 const HeadWeights h, float inv_temp, float* __restrict__ policy, float* __restrict__ winrate,
                 const int* err, int* err_out, uint32_t* run) {
    // a CTA's shared memory may be written from the cluster once that CTA runs: every
    // thread says so here and looks before its first remote store
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    __shared__ float x[3][kHeadCells][kHeadGroup];
    __shared__ float part_pol[2 * kHeadCtas][kMoves];       // of the position this CTA finishes
    __shared__ float part_val[kHeadCtas][kValueHidden];
    __shared__ float scratch[32];
    const int rank = static_cast<int>(head_cluster_rank());
    const int s0 = rank * kHeadCells;
    const int cells = (kSq - s0) < kHeadCells ? (kSq - s0) : kHeadCells;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, warps = kHeadThreads / 32;
    // this thread's plane and output, and its weights
    const int plane = t < kMoves ? 0 : (t < 2 * kMoves ? 1 : 2);
    const int o = t - plane * kMoves;
    const bool owns = plane < 2 || o < kValueHidden;
    const int outs = plane < 2 ? kMoves : kValueHidden;
    const float* wsrc = plane < 2 ? h.ip_pol_wT + (size_t)(plane * kSq + s0) * kMoves + o
                                  : h.ip1_val_wT + (size_t)s0 * kValueHidden + o;
    constexpr int kHeld = kHeadGroup == 1 ? 26 : 18;        // weights held in registers; the rest come from L2 later
    float wr[kHeld];
#pragma unroll
    for (int i = 0; i < kHeld; i++) wr[i] = owns ? wsrc[i * outs] : 0.f;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0 && t == 0) {
        if (err_out != nullptr) *err_out = *err;
        if (run != nullptr) *run += 1u;
    }
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    const int stride = static_cast<int>(gridDim.x / kHeadCtas) * kHeadGroup;
    for (int first = static_cast<int>(blockIdx.x / kHeadCtas) * kHeadGroup; first < n; first += stride) {
        const int group = n - first < kHeadGroup ? n - first : kHeadGroup;
        for (int i = warp; i < cells * group; i += warps) {
            const int g = i / cells, s = i - g * cells;
            const float3 r =
                head_conv_cell<T>(X + head_row<kCells>(first + g, s0 + s) * ldx, w, Cp, lo_off, lo_e5m2, lane);
            if (lane < 3) {
                const float raw = lane == 0 ? r.x : (lane == 1 ? r.y : r.z);
                const float m = lane < 2 ? h.bn_pol_mean[lane] : h.bn_val_mean[0];
                const float is = lane < 2 ? h.bn_pol_invstd[lane] : h.bn_val_invstd[0];
                x[lane][s][g] = fmaxf(nf_mul(is, nf_add(raw, -m)), 0.f);
            }
        }
        __syncthreads();
        if (owns) {
            const float* xp = &x[plane][0][0];
            float acc[kHeadGroup] = {};
#pragma unroll
            for (int i = 0; i < kHeld; i++) {
#pragma unroll
                for (int g = 0; g < kHeadGroup; g++) acc[g] = fmaf(wr[i], xp[i * kHeadGroup + g], acc[g]);
            }
#pragma unroll 7
            for (int i = kHeld; i < cells; i++) {
                const float wv = wsrc[i * outs];
#pragma unroll
                for (int g = 0; g < kHeadGroup; g++) acc[g] = fmaf(wv, xp[i * kHeadGroup + g], acc[g]);
            }
#pragma unroll
            for (int g = 0; g < kHeadGroup; g++) {
                if (plane < 2) store_to_cta(&part_pol[2 * rank + plane][o], g, acc[g]);
                else store_to_cta(&part_val[rank][o], (g + 1) % kHeadCtas, acc[g]);
            }
        }
        __syncthreads();                  // every warp whole again before the aligned cluster barrier
        head_cluster_sync();              // all partial sums have arrived
        if (rank < group) {
            float logit = -INFINITY;
            if (t < kMoves) {
                float acc = 0.f;
#pragma unroll
                for (int k = 0; k < 2 * kHeadCtas; k++) acc += part_pol[k][t];
                logit = h.ip_pol_b[t] + acc;
            }
            const float mx = block_reduce(logit, scratch, true);
            const float e = t < kMoves ? expf((logit - mx) * inv_temp) : 0.f;
            const float denom = block_reduce(e, scratch, false);
            if (t < kMoves) policy[(size_t)(first + rank) * kMoves + t] = e / denom;
        }
        const int vg = (rank + kHeadCtas - 1) % kHeadCtas;      // whose value head this CTA finishes
        if (vg < group) {
            float v = 0.f;
            if (t < kValueHidden) {
                float acc = 0.f;
#pragma unroll
                for (int k = 0; k < kHeadCtas; k++) acc += part_val[k][t];
                v = h.ip2_val_w[t] * fmaxf(h.ip1_val_b[t] + acc, 0.f);
            }
            const float sum = block_reduce(v, scratch, false);
            if (t == 0) winrate[first + vg] = (1.0f + tanhf(h.ip2_val_b[0] + sum)) / 2.0f;
        }
        if (first + stride < n) {
            __syncthreads();
            head_cluster_sync();          // the sums are read: the next group may overwrite them
        }
    }
}

}  // namespace lzb
