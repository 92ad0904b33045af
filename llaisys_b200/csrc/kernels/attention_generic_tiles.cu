// The operator's attention over plain K/V tensors in f32 arithmetic, by tiles: what attention_generic.cu computes with one CTA per (query
// row, head), for one sequence with head_dim 64 or 128 and nothing but the causal mask.
//
// Bound: f32 FMA (two matrix products that must not leave 32 bits). One CTA per row and head read every K and V row once per (row, head),
// lane by lane: 96 rows x 777 keys x 12 heads took 452 us, and the FMAs of it 6 us at the chip's rate. Here a CTA owns kRows rows of one kv
// head -- a row is (query, head of the group), so the heads that share K and V share its tiles -- and walks keys in blocks through shared
// memory with 4 x 4 (4 x 2) scores and 4 x 8 outputs per thread. Keys are split over the CTAs of a cluster, which then exchange (max, sum,
// accumulator) through distributed shared memory: no workspace, no counters, and the order of every sum is fixed. Same call: 43 us, of
// which the shared-memory port is busy for about 30 (an operand read serves four FMAs); one CTA per SM, with the weights beside K instead
// of over it, took 68.
#include "device_utils.cuh"
#include "kernels.hpp"
#include "launch_utils.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace llaisys::kernels {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256, kMostSplits = 8; // (eight CTAs: the largest portable cluster)

struct TileParams {
    const void *q, *k, *v;
    void *out;
    int32_t n_q, total, nh, nkvh; // queries, keys, heads
    float scale;
};

// kRows x kKeys scores per step; warps: kRows / 16 along the rows, the rest along the keys (and along the dims of the output).
template <typename T, int D, int kRows, int kKeys>
struct TileShape {
    static constexpr int kAcross = kThreads / 32 / (kRows / 16);
    static constexpr int kKeysPerLane = kKeys / kAcross / 8;
    static constexpr int kDims = D / kAcross / 8; // output dims of a lane
    static constexpr int kVec = kDims < 4 ? kDims : 4;
    static constexpr int kLd = D + 4, kLdP = kKeys + 4; // rows four words apart in the banks
    static constexpr int kFloats = kRows * kLd + kKeys * kLd + kKeys * D + 3 * kRows;
    static_assert(kRows * kLdP <= kKeys * kLd && kRows <= kKeys, "weights, and at the end accumulators, take the place of K");
};

// Keys [key0, key0 + kKeys) of one kv head -> f32 rows of kLd in shared memory; keys from `end` on become zeros. f32 rows go by cp.async
// (the caller waits), 16-bit rows through registers.
template <typename T, int D, int kKeys, int kLd>
__device__ __forceinline__ void load_keys(float *dst, const T *src, int64_t token_stride, int key0, int end) {
    constexpr int kPer = 16 / sizeof(T), kPieces = kKeys * D / kPer / kThreads;
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int piece = threadIdx.x + i * kThreads, key = piece / (D / kPer), dim = piece % (D / kPer) * kPer;
            const bool live = key0 + key < end;
            const T *from = src + (live ? (key0 + key) * token_stride + dim : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst + key * kLd + dim))),
                         "l"(from), "r"(live ? 16 : 0)
                         : "memory");
        }
    } else {
        uint4 word[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int piece = threadIdx.x + i * kThreads, key = piece / (D / kPer), dim = piece % (D / kPer) * kPer;
            word[i] = key0 + key < end ? *reinterpret_cast<const uint4 *>(src + (key0 + key) * token_stride + dim) : uint4{0, 0, 0, 0};
        }
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int piece = threadIdx.x + i * kThreads, key = piece / (D / kPer), dim = piece % (D / kPer) * kPer;
            const T *in = reinterpret_cast<const T *>(&word[i]);
            float *at = dst + key * kLd + dim;
            *reinterpret_cast<float4 *>(at) = make_float4(to_f32(in[0]), to_f32(in[1]), to_f32(in[2]), to_f32(in[3]));
            *reinterpret_cast<float4 *>(at + 4) = make_float4(to_f32(in[4]), to_f32(in[5]), to_f32(in[6]), to_f32(in[7]));
        }
    }
}

__device__ __forceinline__ void commit_copies() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void wait_copies() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// acc += P V over the block's keys. kCareful: a weight of zero meets no V row (0 x inf and 0 x NaN stay out, as where hidden keys are
// never read).
template <bool kCareful, typename S, int D, int kKeys>
__device__ __forceinline__ void add_values(float (&acc)[4][S::kDims], const float *p_s, const float *v_s, int row0, int dim0, int lane_d) {
    for (int key = 0; key < kKeys; key += 4) {
        float4 p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            p[i] = *reinterpret_cast<const float4 *>(p_s + (row0 + 4 * i) * S::kLdP + key);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v[S::kDims];
#pragma unroll
            for (int n = 0; n < S::kDims / S::kVec; ++n) {
                const float *at = v_s + (key + j) * D + dim0 + (n * 8 + lane_d) * S::kVec;
                if constexpr (S::kVec == 4) {
                    *reinterpret_cast<float4 *>(v + 4 * n) = *reinterpret_cast<const float4 *>(at);
                } else if constexpr (S::kVec == 2) {
                    *reinterpret_cast<float2 *>(v) = *reinterpret_cast<const float2 *>(at);
                } else {
                    v[0] = *at;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float w = j == 0 ? p[i].x : j == 1 ? p[i].y : j == 2 ? p[i].z : p[i].w;
#pragma unroll
                for (int n = 0; n < S::kDims; ++n) {
                    if (!kCareful || w != 0.f) {
                        acc[i][n] = fmaf(w, v[n], acc[i][n]);
                    }
                }
            }
        }
    }
}

template <typename T, int D, int kRows, int kKeys>
__global__ void __launch_bounds__(kThreads, kRows == 64 ? 2 : 1) attention_generic_tiles_kernel(TileParams p) {
    using S = TileShape<T, D, kRows, kKeys>;
    extern __shared__ float4 smem4[];
    float *q_s = reinterpret_cast<float *>(smem4);   // [kRows][kLd], pre-multiplied by scale
    float *k_s = q_s + kRows * S::kLd;               // [kKeys][kLd]; at the end: this CTA's accumulators [kRows][kLd]
    float *v_s = k_s + kKeys * S::kLd;               // [kKeys][D]
    float *p_s = k_s;                                // [kRows][kLdP] scores, then weights, where K was: two CTAs fit an SM
    float *m_s = v_s + kKeys * D, *l_s = m_s + kRows, *a_s = l_s + kRows;

    const cg::cluster_group cluster = cg::this_cluster();
    const int splits = int(cluster.num_blocks()), split = int(cluster.block_rank());
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int group = p.nh / p.nkvh, kvh = blockIdx.y, rows = p.n_q * group, r0 = int(blockIdx.x) / splits * kRows;
    const int before = p.total - p.n_q; // query t sees keys j <= t + before
    const int last = min(r0 + kRows, rows) - 1, limit = before + last / group + 1;
    const int n_blocks = (limit + kKeys - 1) / kKeys;
    const int block0 = int(int64_t(n_blocks) * split / splits), block1 = int(int64_t(n_blocks) * (split + 1) / splits);
    const int64_t token_stride = int64_t(p.nkvh) * D;
    const T *k_base = static_cast<const T *>(p.k) + int64_t(kvh) * D, *v_base = static_cast<const T *>(p.v) + int64_t(kvh) * D;

    if (block0 < block1) {
        load_keys<T, D, kKeys, S::kLd>(k_s, k_base, token_stride, block0 * kKeys, limit);
        commit_copies();
        load_keys<T, D, kKeys, D>(v_s, v_base, token_stride, block0 * kKeys, limit);
        commit_copies();
    }
    constexpr int kPer = 16 / sizeof(T);
#pragma unroll
    for (int i = tid; i < kRows * D / kPer; i += kThreads) {
        const int row = i / (D / kPer), dim = i % (D / kPer) * kPer, r = r0 + row, t = r / group;
        uint4 word{0, 0, 0, 0};
        if (r < rows) {
            word = *reinterpret_cast<const uint4 *>(static_cast<const T *>(p.q) + (int64_t(t) * p.nh + kvh * group + (r - t * group)) * D + dim);
        }
#pragma unroll
        for (int n = 0; n < kPer; ++n) {
            q_s[row * S::kLd + dim + n] = to_f32(reinterpret_cast<const T *>(&word)[n]) * p.scale;
        }
    }
    if (tid < kRows) {
        m_s[tid] = -INFINITY;
        l_s[tid] = 0.f;
    }
    const int warp_r = warp / S::kAcross, warp_c = warp % S::kAcross;
    const int row0 = warp_r * 16 + lane / 8;                                         // rows of a thread: row0 + 4 i
    const int key_lane = warp_c * (kKeys / S::kAcross) + lane % 8;                   // its keys: + 8 j
    const int dim0 = warp_c * (D / S::kAcross);
    const bool idle = r0 + warp_r * 16 >= rows;
    float acc[4][S::kDims];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int n = 0; n < S::kDims; ++n) {
            acc[i][n] = 0.f;
        }
    }

    for (int block = block0; block < block1; ++block) {
        const int key0 = block * kKeys;
        wait_copies<1>(); // K of this block
        __syncthreads();
        float s[4][S::kKeysPerLane];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < S::kKeysPerLane; ++j) {
                s[i][j] = 0.f;
            }
        }
        if (!idle) {
#pragma unroll 4
            for (int dim = 0; dim < D; dim += 4) {
                float4 a[4], b[S::kKeysPerLane];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[i] = *reinterpret_cast<const float4 *>(q_s + (row0 + 4 * i) * S::kLd + dim);
                }
#pragma unroll
                for (int j = 0; j < S::kKeysPerLane; ++j) {
                    b[j] = *reinterpret_cast<const float4 *>(k_s + (key_lane + 8 * j) * S::kLd + dim);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
#pragma unroll
                    for (int j = 0; j < S::kKeysPerLane; ++j) {
                        s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                        s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                        s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                        s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
                    }
                }
            }
        }
        __syncthreads(); // K has been read: the scores go over it
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < S::kKeysPerLane; ++j) {
                p_s[(row0 + 4 * i) * S::kLdP + key_lane + 8 * j] = s[i][j];
            }
        }
        __syncthreads();
        { // softmax: kThreads / kRows neighbouring lanes share a row
            constexpr int kLanes = kThreads / kRows, kEach = kKeys / kLanes;
            const int r = tid / kLanes, part = tid % kLanes;
            const int seen = r0 + r < rows ? before + (r0 + r) / group + 1 - key0 : 0; // of this block's keys
            float *row = p_s + r * S::kLdP;
            float s[kEach], mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < kEach; ++i) {
                s[i] = part + kLanes * i < seen ? row[part + kLanes * i] : -INFINITY;
                mx = fmaxf(mx, s[i]);
            }
#pragma unroll
            for (int o = kLanes / 2; o > 0; o /= 2) {
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            // (fmaxf drops NaN: where nothing but NaN and -inf has been seen the maximum is still -inf, and the weight of a NaN score must
            // come out as NaN; hidden scores are -inf and weigh nothing either way)
            const float m_old = m_s[r], m_new = fmaxf(m_old, mx), base = m_new != -INFINITY ? m_new : 0.f;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < kEach; ++i) {
                const float e = expf(s[i] - base);
                row[part + kLanes * i] = e;
                sum += e;
            }
#pragma unroll
            for (int o = kLanes / 2; o > 0; o /= 2) {
                sum += __shfl_xor_sync(0xffffffffu, sum, o);
            }
            __syncwarp();
            if (part == 0) {
                const float alpha = m_new != -INFINITY ? expf(m_old - m_new) : 1.f;
                a_s[r] = alpha;
                l_s[r] = l_s[r] * alpha + sum;
                m_s[r] = m_new;
            }
        }
        wait_copies<0>(); // V of this block
        int odd = 0;      // a value that a weight of zero must not meet
        for (int i = tid; i < kKeys * D / 4; i += kThreads) {
            const float4 x = reinterpret_cast<const float4 *>(v_s)[i];
            odd |= !(fabsf(x.x) < INFINITY) | !(fabsf(x.y) < INFINITY) | !(fabsf(x.z) < INFINITY) | !(fabsf(x.w) < INFINITY);
        }
        const bool careful = __syncthreads_or(odd) != 0;
        if (!idle) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float alpha = a_s[row0 + 4 * i];
#pragma unroll
                for (int n = 0; n < S::kDims; ++n) {
                    acc[i][n] *= alpha;
                }
            }
            if (careful) {
                add_values<true, S, D, kKeys>(acc, p_s, v_s, row0, dim0, lane % 8);
            } else {
                add_values<false, S, D, kKeys>(acc, p_s, v_s, row0, dim0, lane % 8);
            }
        }
        __syncthreads();
        if (block + 1 < block1) {
            load_keys<T, D, kKeys, S::kLd>(k_s, k_base, token_stride, key0 + kKeys, limit);
        }
        commit_copies();
        if (block + 1 < block1) {
            load_keys<T, D, kKeys, D>(v_s, v_base, token_stride, key0 + kKeys, limit);
        }
        commit_copies();
    }

    // every CTA's accumulators where K was; then each CTA of the cluster finishes its share of the rows
    wait_copies<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int n = 0; n < S::kDims; ++n) {
            k_s[(row0 + 4 * i) * S::kLd + dim0 + (n / S::kVec * 8 + lane % 8) * S::kVec + n % S::kVec] = acc[i][n];
        }
    }
    cluster.sync();
    for (int i = tid; i < kRows / splits * (D / 4); i += kThreads) {
        const int row = split * (kRows / splits) + i / (D / 4), dim = i % (D / 4) * 4, r = r0 + row, t = r / group;
        if (r >= rows) {
            break;
        }
        float m[kMostSplits], m_all = -INFINITY, l_all = 0.f;
        float4 o = {0.f, 0.f, 0.f, 0.f}, part[kMostSplits];
        float l[kMostSplits];
#pragma unroll
        for (int s = 0; s < kMostSplits; ++s) {
            if (s < splits) {
                m[s] = *cluster.map_shared_rank(m_s + row, s);
                l[s] = *cluster.map_shared_rank(l_s + row, s);
                part[s] = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(k_s + row * S::kLd + dim, s));
                m_all = fmaxf(m_all, m[s]);
            }
        }
#pragma unroll
        for (int s = 0; s < kMostSplits; ++s) {
            if (s < splits) {
                const float w = m[s] == -INFINITY ? 0.f : expf(m[s] - m_all); // (0 x NaN: a share of NaN scores alone still shows)
                l_all += l[s] * w;
                o.x += part[s].x * w;
                o.y += part[s].y * w;
                o.z += part[s].z * w;
                o.w += part[s].w * w;
            }
        }
        const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
        T *at = static_cast<T *>(p.out) + (int64_t(t) * p.nh + kvh * group + (r - t * group)) * D + dim;
        at[0] = from_f32<T>(o.x * inv);
        at[1] = from_f32<T>(o.y * inv);
        at[2] = from_f32<T>(o.z * inv);
        at[3] = from_f32<T>(o.w * inv);
    }
    cluster.sync(); // nobody leaves while its shared memory is being read
}

template <typename T, int D, int kRows, int kKeys>
void launch(cudaStream_t s, const TileParams &p, int splits) {
    using S = TileShape<T, D, kRows, kKeys>;
    constexpr int kBytes = S::kFloats * int(sizeof(float));
    auto kernel = attention_generic_tiles_kernel<T, D, kRows, kKeys>;
    LLAISYS_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes));
    cudaLaunchConfig_t cfg{};
    const int tiles = (p.n_q * (p.nh / p.nkvh) + kRows - 1) / kRows;
    cfg.gridDim = dim3(unsigned(tiles * splits), unsigned(p.nkvh));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(splits);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LLAISYS_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, p));
}

template <typename T>
void dispatch(cudaStream_t s, const TileParams &p, int d) {
    // Few rows: tiles of 16, so that the rows spread over the chip (at 64 a tile's row count would be padding, or a handful of CTAs would
    // do all of the work); a cluster of up to eight CTAs per tile while the grid is small and there are keys to split. 12 / 2 heads of 128,
    // f32, 400 keys, by row and head and in tiles: 1 query 62 and 13 us, 16 queries 88 and 15, 40 queries 137 and 15.
    const int64_t rows = int64_t(p.n_q) * (p.nh / p.nkvh);
    const int64_t few = (rows + 15) / 16 * p.nkvh, many = (rows + 63) / 64 * p.nkvh;
    const bool small = few <= 64;
    const int blocks = (p.total + (small ? 127 : 63)) / (small ? 128 : 64);
    int splits = 1;
    // (never fewer than four CTAs where there are keys for them: a sum over 1600 keys in one piece is off by 5.7e-7 where four are by 4.9e-7)
    while (splits < kMostSplits && splits < blocks && (splits < 4 || (small ? few : many) * splits < device_sms())) {
        splits *= 2;
    }
    if (d == 128) {
        small ? launch<T, 128, 16, 128>(s, p, splits) : launch<T, 128, 64, 64>(s, p, splits);
    } else {
        small ? launch<T, 64, 16, 128>(s, p, splits) : launch<T, 64, 64, 64>(s, p, splits);
    }
}

} // namespace

bool attention_generic_tiles(stream_t stream, llaisysDataType_t dtype, const KVView &kv, const AttnBatch &batch, const void *q, float scale,
                             const AttnOut &out) {
    const bool plain = kv.block_table == nullptr && batch.n_seqs == 1 && batch.q_starts == nullptr && batch.kv_lens == nullptr &&
                       batch.window <= 0 && batch.fade_a == nullptr && out.out != nullptr && out.part == nullptr && out.row_scale == nullptr &&
                       out.row_stride == 0 && kv.vDim() == kv.d && (kv.d == 64 || kv.d == 128) && kv.head_stride == kv.d &&
                       kv.token_stride == int64_t(kv.nkvh) * kv.d && kv.page_stride == kv.page_size * kv.token_stride;
    auto aligned = [](const void *ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0; }; // q, K and V come in pieces of 16 bytes
    // Up to 16 keys a tile is mostly padding and the cluster's start-up is the call. One CTA per (row, head) takes 6.5, 8.7 and 10.7 us for 4, 8
    // and 16 keys with heads of 64, 8.7, 10.7 and 12.8 with heads of 128; tiles take 10.7 and 12.8 to 14.8 up to 32 keys, where the other
    // kernel is at 15 and 18.
    constexpr int kFewKeys = 16;
    if (!plain || !aligned(q) || !aligned(kv.k_base) || !aligned(kv.v_base) || kv.nkvh > 65535 || batch.total_q != batch.const_q_len ||
        batch.const_kv_len < batch.const_q_len || batch.const_kv_len <= kFewKeys || int64_t(batch.total_q) * (batch.nh / kv.nkvh) > (int64_t(1) << 27)) {
        return false;
    }
    const TileParams p{q, kv.k_base, kv.v_base, out.out, batch.total_q, batch.const_kv_len, batch.nh, kv.nkvh, scale};
    auto s = static_cast<cudaStream_t>(stream);
    switch (dtype) {
    case LLAISYS_DTYPE_F32:
        dispatch<float>(s, p, kv.d);
        return true;
    case LLAISYS_DTYPE_F16:
        dispatch<__half>(s, p, kv.d);
        return true;
    case LLAISYS_DTYPE_BF16:
        dispatch<__nv_bfloat16>(s, p, kv.d);
        return true;
    default:
        return false;
    }
}

} // namespace llaisys::kernels
