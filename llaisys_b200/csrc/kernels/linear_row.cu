// One row of activations through a 16-bit weight matrix, with what stands around it in a decoder block: out = f(x) . W^T with f the RMS norm
// or nothing, and the sums stored, added to a residual row, or -- W a packed gate|up matrix -- gated.
//
// Bound: HBM, every weight is read once (2 flops a byte). A GEMM call for one row is a launch that starts cold behind the norm's launch: for
// a width of 1536 the norm, the 2048-row projection, the 17920-row one and its activation, and the 8960-deep one took 3.5, 6.4, 11 + 2 and
// 12.8 us, of which the bytes are 1, 8.5 and 4.3. Here a warp owns two rows of W (a gate row and its up row) and keeps up to twelve 16-byte
// loads in flight; where K is deep eight warps share two rows. The launch is programmatic and the first loads of W are issued BEFORE the wait
// for the kernel in front (weights are not written by kernels), so the stream of weights does not stop between the launches of a step; each
// CTA normalises the row itself. Products and sums are f32, f(x) is rounded to 16 bits as the separate norm rounds it.
// One token through four layers and a vocabulary of 32768, steps queued in a row, us before -> now (time of the weights' bytes alone): width 896
// / 4864 243 -> 193 (30), 1536 / 8960 298 -> 226 (74), 2048 / 5632 345 -> 235 (75), 4096 / 14336 670 -> 508 (312), 5120 / 13824 754 -> 659
// (393), 8192 / 28672 1504 -> 1423 (1144); depths over kMostK (14336 up) stay with the general path in these.
#include "launch_utils.cuh"
#include "mma_utils.cuh"

#include <algorithm>

namespace llaisys::kernels {

namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kLoads = 6;     // 16-byte pieces of a row that a lane holds at a time
constexpr int kMostK = 12000; // f(x) as f32 within 48 KiB of shared memory

struct RowArgs {
    void *out;
    const void *x, *gain, *w; // gain null: no norm
    float eps;
    int32_t n, k;      // outputs, depth
    int32_t ways;      // warps that share a row pair: 1 or 8
    int32_t glu, add;  // rows g and n + g of W make output g; out += instead of out =
};

template <typename T>
__global__ void __launch_bounds__(kThreads, 2) linear_row_kernel(RowArgs a) {
    extern __shared__ float4 x_s[]; // f(x): the first four elements of every piece, then the last four
    __shared__ float s_norm[kWarps], s_part[kWarps][2];
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int pieces = a.k / 8, per_cta = kWarps / a.ways, way = warp % a.ways;
    const int groups = a.glu ? a.n : (a.n + 1) / 2;
    const int chunks = (pieces + kLoads * 32 * a.ways - 1) / (kLoads * 32 * a.ways);
    auto row_of = [&](int g, int r) { return a.glu ? g + r * a.n : 2 * g + r; };

    uint4 held[2][kLoads];
    auto load = [&](int g, int c) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool live = g < groups && (a.glu || 2 * g + r < a.n);
            const uint4 *row = static_cast<const uint4 *>(a.w) + int64_t(live ? row_of(g, r) : 0) * pieces;
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                const int piece = ((c * kLoads + u) * a.ways + way) * 32 + lane;
                held[r][u] = make_uint4(0u, 0u, 0u, 0u);
                if (live && piece < pieces) {
                    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(held[r][u].x), "=r"(held[r][u].y), "=r"(held[r][u].z), "=r"(held[r][u].w)
                                 : "l"(row + piece));
                }
            }
        }
    };
    int g = blockIdx.x * per_cta + warp / a.ways;
    load(g, 0);
    grid_dependency_wait();
    grid_launch_dependents();

    float inv = 1.f;
    const uint4 *x = static_cast<const uint4 *>(a.x);
    if (a.gain != nullptr) {
        float ss = 0.f;
        for (int i = tid; i < pieces; i += kThreads) {
            const uint4 word = x[i];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float v = to_f32(reinterpret_cast<const T *>(&word)[e]);
                ss = fmaf(v, v, ss);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o /= 2) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        }
        if (lane == 0) {
            s_norm[warp] = ss;
        }
        __syncthreads();
        float total = 0.f;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) {
            total += s_norm[i];
        }
        inv = rsqrtf(total / float(a.k) + a.eps);
    }
    for (int i = tid; i < pieces; i += kThreads) {
        const uint4 word = x[i], gain = a.gain != nullptr ? static_cast<const uint4 *>(a.gain)[i] : uint4{};
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = to_f32(reinterpret_cast<const T *>(&word)[e]);
            if (a.gain != nullptr) {
                v[e] = to_f32(from_f32<T>(to_f32(reinterpret_cast<const T *>(&gain)[e]) * v[e] * inv));
            }
        }
        x_s[i] = make_float4(v[0], v[1], v[2], v[3]);
        x_s[pieces + i] = make_float4(v[4], v[5], v[6], v[7]);
    }
    __syncthreads();

    // (eight warps on a pair: g is the CTA's, so the barriers below meet)
    for (; g < groups; g += int(gridDim.x) * per_cta) {
        float sum[2] = {0.f, 0.f};
        for (int c = 0; c < chunks; ++c) {
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                const int piece = ((c * kLoads + u) * a.ways + way) * 32 + lane;
                if (piece < pieces) {
                    const float4 lo = x_s[piece], hi = x_s[pieces + piece];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const T *w = reinterpret_cast<const T *>(&held[r][u]);
                        sum[r] = fmaf(lo.x, to_f32(w[0]), sum[r]);
                        sum[r] = fmaf(lo.y, to_f32(w[1]), sum[r]);
                        sum[r] = fmaf(lo.z, to_f32(w[2]), sum[r]);
                        sum[r] = fmaf(lo.w, to_f32(w[3]), sum[r]);
                        sum[r] = fmaf(hi.x, to_f32(w[4]), sum[r]);
                        sum[r] = fmaf(hi.y, to_f32(w[5]), sum[r]);
                        sum[r] = fmaf(hi.z, to_f32(w[6]), sum[r]);
                        sum[r] = fmaf(hi.w, to_f32(w[7]), sum[r]);
                    }
                }
            }
            c + 1 < chunks ? load(g, c + 1) : load(g + int(gridDim.x) * per_cta, 0);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int o = 16; o > 0; o /= 2) {
                sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
            }
        }
        if (a.ways > 1) {
            if (lane == 0) {
                s_part[warp][0] = sum[0];
                s_part[warp][1] = sum[1];
            }
            __syncthreads();
            sum[0] = sum[1] = 0.f;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) {
                sum[0] += s_part[i][0];
                sum[1] += s_part[i][1];
            }
            __syncthreads();
        }
        if (way == 0 && lane == 0) {
            T *out = static_cast<T *>(a.out);
            if (a.glu) {
                out[g] = from_f32<T>(sum[1] * (sum[0] / (1.f + expf(-sum[0]))));
            } else {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (2 * g + r < a.n) {
                        out[2 * g + r] = from_f32<T>(a.add ? to_f32(out[2 * g + r]) + sum[r] : sum[r]);
                    }
                }
            }
        }
    }
}

} // namespace

bool linear_row(stream_t stream, llaisysDataType_t dtype, void *out, const void *x, const void *gain, float eps, const void *weight, size_t n,
                size_t k, RowOut form) {
    if ((dtype != LLAISYS_DTYPE_BF16 && dtype != LLAISYS_DTYPE_F16) || n == 0 || n > (size_t(1) << 30) || k == 0 || k % 8 != 0 || k > kMostK ||
        !aligned16(x) || !aligned16(weight) || (gain != nullptr && !aligned16(gain)) || linear_policy() != 0) {
        return false;
    }
    RowArgs a{out, x, gain, weight, eps, int32_t(n), int32_t(k), 0, form == RowOut::kGlu, form == RowOut::kAdd};
    // Rows of up to 12 KiB go through a warp in a few loads; behind that the few rows of a deep matrix (1536 of 8960) would leave the chip with
    // five warps an SM, so a CTA shares them. (The line was not swept; layers with depths of 5632 to 8192 on either side gain alike, see above.)
    a.ways = k > 6144 ? kWarps : 1;
    const size_t groups = form == RowOut::kGlu ? n : (n + 1) / 2, per_cta = size_t(kWarps / a.ways);
    const unsigned grid = unsigned(std::min<size_t>((groups + per_cta - 1) / per_cta, size_t(device_sms()) * 2)); // (two CTAs fit an SM)
    auto s = static_cast<cudaStream_t>(stream);
    if (dtype == LLAISYS_DTYPE_BF16) {
        launch_programmatic_smem(linear_row_kernel<__nv_bfloat16>, grid, kThreads, k * sizeof(float), s, a);
    } else {
        launch_programmatic_smem(linear_row_kernel<__half>, grid, kThreads, k * sizeof(float), s, a);
    }
    check_launch("linear_row");
    return true;
}

} // namespace llaisys::kernels
