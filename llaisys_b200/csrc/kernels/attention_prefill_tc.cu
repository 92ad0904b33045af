// K4: attention of chunks of new tokens over the page pool (and over the operator's plain K/V tensors) on the 5th-generation tensor
// cores: tcgen05.mma, operands by TMA, scores, weights and accumulators in tensor memory.
//
// Bound: the tensor pipe and, at the same rate, the exponentials: a block of 256 rows x 128 keys is 2048 clocks of MMA on an SM and 2048
// clocks of ex2 (16 a clock). Bytes are no bound: K and V of a block are 64 KiB per 2048 clocks.
//
// Work. A ROW is (query, head of the group): the heads that share a kv head share its K and V, so rows are packed over queries and heads
// and a TILE is (sequence, 256 packed rows, kv head). Tiles of 128 queries of one head, as before, filled a chunk of 20 tokens to a sixth
// and fetched K and V once per head. A tile visits its visible keys 128 at a time (a BLOCK: 8 pages). All blocks of all tiles, in the order
// (sequence, row block, kv head, key block), form one line that is cut into equal pieces, one per SM, so that every SM gets the same number
// of blocks whatever the mix of lengths; where tiles are short, whole tiles are dealt out instead. A piece covers the end of one tile,
// whole tiles, and the beginning of another; each such FRAGMENT runs like a tile. A fragment that is its whole tile normalises and stores
// its rows; otherwise it stores the accumulator and the rows' (max, sum) into a slot of a workspace and counts itself in, and the fragment
// that arrives last merges the others with what it holds, in the order of the CTAs and not of arrival. Nobody waits for another CTA.
//
// Per CTA (one per SM):
//   warp 8   reads the block table and issues TMA tiles (16 tokens x 64 dims, 128-byte swizzle) into a ring of five 32 KiB stages, K and V of
//            a block in turn, across fragment boundaries;
//   warps 9, 10   issue the MMAs of the tile's two halves of 128 rows, [P V of block i, Q K^T of block i + 1] at a time, in turn: the pipe
//            works on one half while the other half's softmax runs;
//   warps 0-3, 4-7   softmax of half 0 and half 1, one row per thread (its tensor memory lane): scores to registers, running maximum,
//            P = 2^(s - m) as 16-bit pairs over the scores' columns in two parts (the product starts on the first while the second is
//            computed), the accumulator rescaled only when a row's maximum grew by more than 2^8.
// Tensor memory: 2 x 128 columns of scores, 2 x 128 of accumulators: all 512. Shared memory: Q 64 KiB, ring 160 KiB.
//
// Tiles of 128 rows of one head on two CTAs per SM (attention_narrow_tc.cu, which took all of these calls before) have twice the barriers,
// commits and TMA boxes per score, and Q K^T at N 64 bound by the shared-memory port. Append and attention of a layer, narrow and here, many in
// a row: a prompt of 8192 tokens, 32 / 8 heads 618 and 545 us; 8 chunks of 512 behind up to 8192 tokens, 12 / 2 heads 142 and 127; 24 pieces of
// 1 to 96 tokens behind up to 3000 55 and 40; 3 of 1500 to 4000 with a window of 1024, 32 / 8 heads 285 and 210. A block takes a CTA about 3000
// clocks: a half's chain of scores to registers (250), maximum (350), exponentials (2 x 650) and its MMAs (1024) is what is left above 2048.
//
// Synchronisation is mbarriers only (and a named barrier per half around the arrival count). Every wait is bounded: one that runs out sets
// bit 8 of the error word, nothing is issued or loaded behind it, and the others give up at their next wait. Whatever way a role ends, it sees
// its own MMAs or copies done before the CTA gives its tensor memory back and leaves. No cluster launch, no multicast.
#include "kernels.hpp"
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace llaisys::kernels {

namespace {

constexpr int kD = 128, kPage = 16;
constexpr int kHalf = 128, kRows = 2 * kHalf; // packed rows of a half and of a tile
constexpr int kKeys = 128, kPagesPerBlock = kKeys / kPage;
constexpr int kStages = 5, kStageBytes = kKeys * kD * 2, kPieceBytes = kKeys * 128; // a stage: K or V of a block; K: [dims 0-63 | 64-127][128 keys][128 B]
constexpr int kQBytes = kHalf * kD * 2, kQPiece = kHalf * 128;                       // per half: [dims 0-63 | 64-127][128 rows][128 B]
constexpr int kSoftmaxThreads = 128, kProducerWarp = 8, kMmaWarp = 9, kThreads = 384;
// Registers a thread: 384 x 168 at launch, then 256 softmax threads take 224 and the 128 of the other four warps (one of them idle) keep 56.
constexpr int kSoftmaxRegs = 224, kOtherRegs = 56;
static_assert(256 * kSoftmaxRegs + 128 * kOtherRegs <= kThreads * 168, "no more than the CTA was launched with");
constexpr int kSchedInts = 44; // sums, maxima and tiles of twelve warps; start of the piece, arrivals, the piece
constexpr int kPlaceInts = 25; // words of shared memory in which a warp keeps its place on the line
constexpr int kTmemCols = 512, kColS = 0, kColO = 2 * kKeys; // scores of half h at kColS + 128 h, accumulators at kColO + 128 h
constexpr int kErrTimeout = 8;
constexpr float kRescaleThreshold = 8.f; // log2 units
// One half's partial result: the accumulator as float4 [32 dim-quads][128 rows], then the rows' maxima and sums.
constexpr int kPartialFloats = kHalf * kD + 2 * kHalf;
// Merging a partial costs its reader about as much as kMergeCostBlocks blocks; shorter pieces than sqrt(kMergeCostBlocks * longest tile)
// would spend more on merging than they save.
constexpr float kMergeCostBlocks = 1.5f;
constexpr int kMergeCost = 5; // (of a tile in two or three pieces: eight blocks whole take 2 us less than in pieces of five units, twelve 3 us more)
// What a tile costs besides its blocks (loading Q, draining the pipeline, storing its rows: about 11500 clocks), in units of a block's time.
constexpr int kTileCost = 4;

enum : int {
    kBarFull = 0,                    // [kStages] producer -> MMA: the stage has landed (transaction bytes)
    // (ONE tcgen05.commit per batch of MMAs; softmax threads, who have seen the batch done, free its stages)
    kBarEmpty = kBarFull + kStages,  // [kStages] softmax (one thread per half; issuer of a half without rows) -> producer: the stage has been read
    kBarS = kBarEmpty + kStages,     // [2] MMA (commit) -> softmax of a half: [P V of the block before, Q K^T of this one] are done
    kBarO = kBarS + 2,               // [2] MMA (commit) -> softmax: the last product of the fragment is done (a barrier of its own: the next
                                     // fragment's first scores may be there before every thread has seen it)
    kBarTurn = kBarO + 2,            // [2] issuer of the other half -> issuer of this half: its batch is issued, the next one is yours
    kBarDrain = kBarTurn + 2,        // [2] MMA (commit) -> the issuer itself: everything it issued has finished
    kBarP = kBarDrain + 2,           // [2][2] softmax (128) -> MMA: this part of P is in tensor memory (and the accumulator rescaled)
    kBarQ = kBarP + 4,               // [2] softmax (128) -> MMA: the next fragment's Q rows are in shared memory
    kNumBars = kBarQ + 2
};
constexpr size_t kSmemBytes = 1024 + 2 * size_t(kQBytes) + kStages * size_t(kStageBytes) + kNumBars * 8 + 8 + kSchedInts * sizeof(int) +
                              kThreads / 32 * kPlaceInts * sizeof(int);
static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");

struct ChunkParams {
    long long page0;
    const int32_t *block_table;
    int32_t table_stride, num_pages;
    const int32_t *seq_ids, *kv_lens, *q_starts; // q_starts [n_seqs + 1]; null in contiguous mode
    int32_t contiguous; // 1: K and V are plain [tokens, nkvh, 128] tensors of ONE sequence; q rows [0, const_q_len), const_kv_len keys
    int32_t const_q_len, const_kv_len;
    int32_t n_seqs, nkvh, group, nh;
    uint32_t group_inverse; // ceil(2^32 / group): x / group = umulhi(x, .) for x < 2^29 (group 1: taken apart)
    const void *q;
    void *out;
    float scale_log2;
    int32_t *error_flag;
    float *partials;   // [gridDim.x][tile begins here: 0, 1][half][kPartialFloats]
    int32_t *counters; // [gridDim.x][half], zero between launches
    // windowed instantiation: query t sees keys j > t + off - window and j < keep_first; row_scale (null: 1) multiplies (row, head)
    int32_t window, keep_first;
    long long out_stride; // elements between rows of out
    const float *row_scale;
    const float *fade_a, *fade_b; // fading instantiation: fade_a[h] log2(1 + fade_b[h] (distance)) is taken off the scores in the log2 domain
    uint32_t wait_limit;          // polls before a wait gives up, where not kMbarWaitLimit
    int32_t out_wide;             // out is 32-byte aligned: rows are stored 32 bytes (a whole sector) per instruction
};

// ---- the line of blocks ------------------------------------------------------------------------------------------

struct SeqGeom {
    int q_start, q_len, kv_len, off, n_qb; // query t sees keys j <= t + off
    int group, window, kept_blocks;        // window 0: none; kept_blocks: blocks that hold the first tokens a window keeps
};

__device__ __forceinline__ SeqGeom seq_geom(const ChunkParams &p, int a) {
    SeqGeom g;
    if (p.contiguous) {
        g.q_start = 0;
        g.q_len = p.const_q_len;
        g.kv_len = max(p.const_kv_len, g.q_len);
    } else {
        g.q_start = p.q_starts[a];
        g.q_len = p.q_starts[a + 1] - g.q_start;
        g.kv_len = min(max(p.kv_lens[a], g.q_len), p.table_stride * kPage);
    }
    g.q_len = min(g.q_len, g.kv_len); // (a chunk longer than the tables can hold: flagged elsewhere, never off the end here)
    g.off = g.kv_len - g.q_len;
    g.n_qb = (g.q_len * p.group + kRows - 1) / kRows;
    g.group = p.group;
    g.window = p.window;
    g.kept_blocks = (p.keep_first + kKeys - 1) / kKeys;
    return g;
}

// keys any row of row block qb can see
__device__ __forceinline__ int tile_kv_hi(const SeqGeom &g, int qb) { return min(g.kv_len, (qb * kRows + kRows - 1) / g.group + 1 + g.off); }
// key blocks that no row of the row block sees, between the blocks of the kept first tokens and the one where the window of its first
// row begins; a tile's blocks are counted without them
__device__ __forceinline__ int tile_gap(const SeqGeom &g, int qb) {
    return g.window > 0 ? max(qb * kRows / g.group + g.off - g.window + 1 - g.kept_blocks * kKeys, 0) / kKeys : 0;
}
__device__ __forceinline__ int tile_blocks(const SeqGeom &g, int qb) { return (tile_kv_hi(g, qb) + kKeys - 1) / kKeys - tile_gap(g, qb); }

// sum of floor((2 i + b) / m) over i < n, for 0 <= b and m <= 8
__device__ __forceinline__ int floor_sum(int n, int m, int b) {
    int sum = 0, a = 2;
    while (n > 0) {
        sum += n * (n - 1) / 2 * (a / m) + n * (b / m);
        a %= m;
        b %= m;
        const int y = a * n + b;
        if (y < m) {
            break;
        }
        n = y / m;
        b = y % m;
        const int t = m;
        m = a;
        a = t;
    }
    return sum;
}
// Units of the line in front of row block qb of a sequence (qb < n_qb), per kv head. Whole tiles: one each. Else the tiles' blocks in closed
// form -- tile i ends at key floor((256 i + 255) / group) + 1 + off, so it has floor((2 i + B) / group) blocks, and its gap is such a term too -- and kTileCost each
__device__ __forceinline__ int units_before(const SeqGeom &g, int qb, bool whole) {
    static_assert(kRows == 2 * kKeys, "row blocks advance two key blocks over the group's heads");
    if (whole) {
        return qb;
    }
    int units = qb * kTileCost + floor_sum(qb, g.group, (kRows - 1 + g.group * (g.off + kKeys)) >> 7);
    if (g.window > 0) {
        const int c = g.group * (g.off - g.window + 1 - g.kept_blocks * kKeys), q0 = c >= 0 ? 0 : (-c + kRows - 1) / kRows;
        if (q0 < qb) {
            units -= floor_sum(qb - q0, g.group, 2 * q0 + (c >> 7)); // (an arithmetic shift: floor)
        }
    }
    return units;
}
// units of a whole sequence
__device__ __forceinline__ int seq_units(const ChunkParams &p, const SeqGeom &g, bool whole) {
    if (whole || g.n_qb == 0) {
        return g.n_qb * p.nkvh;
    }
    return (units_before(g, g.n_qb - 1, false) + tile_blocks(g, g.n_qb - 1) + kTileCost) * p.nkvh;
}

// Position on the line: every role of the CTA walks the same fragments with one of these.
struct Walker {
    int a;         // sequence
    int seq_begin; // index on the line of its first unit
    int n_units;   // its units (all kv heads)
    SeqGeom g;
    int qb, qb_begin; // the row block of the last position asked for, and its first unit inside the sequence (positions only move forward)
    bool whole;       // a unit is a whole tile
};

struct Fragment {
    int a, qb, kvh;
    int b0, b1;     // key blocks [b0, b1) of the tile, counted without its gap
    int gap;        // tile_gap
    int tile_nblk;  // blocks of the whole tile
    int tile_begin; // index on the line of the tile's block 0
    int rows;       // live rows of the tile
    int units;      // from its first unit to the position behind it
};
struct Place {
    Walker w;
    Fragment f;
    int pos; // on the line, behind the fragment
};
static_assert(sizeof(Place) <= kPlaceInts * sizeof(int), "a warp's words");

// The fragment that starts at or after unit `pos` of the line and before piece_end: `pos` moves on to its first block (over the units
// at a tile's end that stand for no block). False when the piece holds no further block.
__device__ __forceinline__ bool locate(const ChunkParams &p, Walker &w, int &pos, int piece_end, Fragment &f) {
    while (pos < piece_end) {
        while (pos >= w.seq_begin + w.n_units && w.a + 1 < p.n_seqs) {
            w.seq_begin += w.n_units;
            ++w.a;
            w.g = seq_geom(p, w.a);
            w.n_units = seq_units(p, w.g, w.whole);
            w.qb = w.qb_begin = 0;
        }
        int x = pos - w.seq_begin - w.qb_begin, nb = tile_blocks(w.g, w.qb), span = w.whole ? 1 : nb + kTileCost;
        while (x >= span * p.nkvh && w.qb + 1 < w.g.n_qb) {
            x -= span * p.nkvh;
            w.qb_begin += span * p.nkvh;
            nb = tile_blocks(w.g, ++w.qb);
            span = w.whole ? 1 : nb + kTileCost;
        }
        const int kvh = min(x / span, p.nkvh - 1), b0 = x - kvh * span;
        if (b0 >= span) {
            return false; // (past the end of the line: no caller asks)
        }
        if (b0 >= nb) { // behind the tile's last block: on to the next tile
            pos += span - b0;
            continue;
        }
        f.a = w.a;
        f.qb = w.qb;
        f.kvh = kvh;
        f.b0 = b0;
        f.tile_nblk = nb;
        f.gap = tile_gap(w.g, w.qb);
        f.b1 = w.whole ? nb : min(nb, b0 + (piece_end - pos));
        f.units = w.whole ? 1 : f.b1 - b0;
        f.tile_begin = pos - b0;
        f.rows = min(kRows, w.g.q_len * w.g.group - w.qb * kRows);
        return true;
    }
    return false;
}

// Blackwell's wider scalar arithmetic for the softmax rows: a three-input maximum and two-wide f32 multiply-add / add
// (one instruction for two scores: these warps are short of issue slots, not of pipe throughput).
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ void fma2(float &x0, float &x1, float a0, float a1, float b, float c) { // x = a * b + c
    asm("{\n"
        ".reg .b64 ra, rb, rc, rd;\n"
        "mov.b64 ra, {%2, %3};\n"
        "mov.b64 rb, {%4, %4};\n"
        "mov.b64 rc, {%5, %5};\n"
        "fma.rn.f32x2 rd, ra, rb, rc;\n"
        "mov.b64 {%0, %1}, rd;\n"
        "}\n"
        : "=f"(x0), "=f"(x1)
        : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void add2(float &s0, float &s1, float a0, float a1) { // s += a
    asm("{\n"
        ".reg .b64 rs, ra;\n"
        "mov.b64 rs, {%0, %1};\n"
        "mov.b64 ra, {%2, %3};\n"
        "add.rn.f32x2 rs, rs, ra;\n"
        "mov.b64 {%0, %1}, rs;\n"
        "}\n"
        : "+f"(s0), "+f"(s1)
        : "f"(a0), "f"(a1));
}

template <bool kBf16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
    if constexpr (kBf16) {
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    } else {
        return __half22float2(*reinterpret_cast<const __half2 *>(&w));
    }
}

// What an instantiation of the kernel adds to plain causal attention; the plain kernel's loops carry nothing of it.
enum Form {
    kPlain,
    kWindowed, // sliding window, output row stride and output factor
    kFading,   // the same with a distance penalty
};

template <bool kBf16, int kForm, bool kShortWaits>
__global__ void __launch_bounds__(kThreads, 1)
    paged_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmap_v, ChunkParams p) {
    constexpr bool kWin = kForm != kPlain, kFade = kForm == kFading;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw_u32 = smem_u32(smem_raw);
    const uint32_t base_u32 = (raw_u32 + 1023u) & ~1023u; // swizzled operands need 1 KiB alignment
    unsigned char *base = smem_raw + (base_u32 - raw_u32);
    const uint32_t ring_u32 = base_u32 + 2 * kQBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + 2 * kQBytes + kStages * kStageBytes);
    const uint32_t bars_u32 = smem_u32(bars);
    uint32_t *s_tmem_base = reinterpret_cast<uint32_t *>(bars + kNumBars);
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem_base + 1);
    int *s_sched = reinterpret_cast<int *>(s_tmem_base + 2); // [kSchedInts]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kWarps = kThreads / 32;

    // ---- this CTA's piece of the line ----------------------------------------------------------------------------
    // (every CTA sums the sequences' units itself: a few loads per sequence, no launch in front of this one)
    int line_units = 0, longest_tile = 0, tiles = 0;
    {
        int mine = 0, mine_max = 0, mine_tiles = 0;
        for (int a = tid; a < p.n_seqs; a += kThreads) {
            const SeqGeom g = seq_geom(p, a);
            mine += seq_units(p, g, false);
            mine_tiles += seq_units(p, g, true);
            // (with a window: what a tile can reach, it only sizes the pieces)
            const int reach = g.window > 0 ? (g.window + kRows / g.group + kKeys) / kKeys + 1 + g.kept_blocks : 1 << 30;
            mine_max = max(mine_max, g.n_qb > 0 ? min((g.kv_len + kKeys - 1) / kKeys, reach) : 0);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            mine += __shfl_xor_sync(0xffffffffu, mine, d);
            mine_max = max(mine_max, __shfl_xor_sync(0xffffffffu, mine_max, d));
            mine_tiles += __shfl_xor_sync(0xffffffffu, mine_tiles, d);
        }
        if (lane == 0) {
            s_sched[warp] = mine;
            s_sched[kWarps + warp] = mine_max;
            s_sched[2 * kWarps + warp] = mine_tiles;
        }
        __syncthreads();
        for (int w = 0; w < kWarps; ++w) {
            line_units += s_sched[w];
            longest_tile = max(longest_tile, s_sched[kWarps + w]);
            tiles += s_sched[2 * kWarps + w];
        }
    }
    const int n_slots = int(gridDim.x);
    const int min_piece = int(ceilf(sqrtf(kMergeCostBlocks * float(longest_tile))));
    int piece = max((line_units + n_slots - 1) / n_slots, max(min_piece, kTileCost + 1)); // units per CTA
    // A cut costs its second CTA what a tile costs, and the merge: where no CTA has more to do with whole tiles alone, there are no cuts.
    // (24 chunks of 100 tokens behind 200, 12 / 2 heads, are 144 tiles of three blocks: cut into equal pieces nearly every CTA had parts of two
    // tiles, 35 us a layer; whole 22.)
    const int tiles_each = (tiles + n_slots - 1) / n_slots;
    const bool whole = (long long)tiles_each * (longest_tile + kTileCost) <= piece + kTileCost + kMergeCost;
    if (whole) {
        piece = tiles_each;
        line_units = tiles;
    }
    const int slot = int(blockIdx.x);
    const int piece_begin = slot * piece;
    if (piece_begin >= line_units) {
        return; // uniform over the CTA, before any mbarrier or TMEM allocation
    }
    const int piece_end = min(line_units, piece_begin + piece);
    volatile int *s_line = s_sched + 3 * kWarps + 4; // units per piece, end of this one (kept there for the same reason as a warp's place)
    if (tid == 0) {
        s_line[0] = piece;
        s_line[1] = piece_end;
    }
    {
        // the sequence that holds unit piece_begin, by a block-wide scan over kThreads sequences at a time
        __syncthreads();
        int before = 0; // units of the sequences in front of this pass's
        for (int a0 = 0; a0 < p.n_seqs; a0 += kThreads) {
            const int a = a0 + tid;
            const int w_a = a < p.n_seqs ? seq_units(p, seq_geom(p, a), whole) : 0;
            int incl = w_a;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, d);
                incl += lane >= d ? up : 0;
            }
            if (lane == 31) {
                s_sched[warp] = incl;
            }
            __syncthreads();
            int warps_before = 0, round_total = 0;
            for (int w = 0; w < kWarps; ++w) {
                warps_before += w < warp ? s_sched[w] : 0;
                round_total += s_sched[w];
            }
            const int excl = before + warps_before + incl - w_a;
            if (w_a > 0 && excl <= piece_begin && piece_begin < excl + w_a) {
                s_sched[3 * kWarps] = a;
                s_sched[3 * kWarps + 1] = excl;
            }
            before += round_total;
            __syncthreads();
            if (before > piece_begin) {
                break;
            }
        }
    }
    Walker walker;
    walker.a = s_sched[3 * kWarps];
    walker.seq_begin = s_sched[3 * kWarps + 1];
    walker.g = seq_geom(p, walker.a);
    walker.whole = whole;
    walker.n_units = seq_units(p, walker.g, whole);
    {
        // the last row block that starts at or before the piece: by bisection, a long chunk has hundreds
        int lo = 0, hi = walker.g.n_qb - 1;
        const int at = piece_begin - walker.seq_begin;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (units_before(walker.g, mid, whole) * p.nkvh <= at) {
                lo = mid;
            } else {
                hi = mid - 1;
            }
        }
        walker.qb = lo;
        walker.qb_begin = units_before(walker.g, lo, whole) * p.nkvh;
    }
    {
        Walker first = walker;
        Fragment f;
        int pos0 = piece_begin;
        if (!locate(p, first, pos0, piece_end, f)) {
            return; // the piece holds no block (the line's last units): uniform over the CTA, nothing set up yet
        }
    }

    // ---- set-up: barriers, TMEM ----------------------------------------------------------------------------------
    if (tid == 0) {
        for (int i = 0; i < kNumBars; ++i) {
            mbar_init(bars_u32 + i * 8, i >= kBarP ? kSoftmaxThreads : i >= kBarEmpty && i < kBarS ? 2 : 1);
        }
        *s_abort = 0;
        mbar_init_fence();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(s_tmem_base), kTmemCols);
        tmem_relinquish();
    }
    // Everything above read only the launch's index arrays and set up on-chip state; q, the K/V rows of the chunk, the workspace and
    // the outputs belong to the stream's order: with launch overlap on, wait here for the kernel directly before this one, and only then
    // let the one behind this one start.
    grid_dependency_wait();
    grid_launch_dependents();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem_base;

    auto bar = [&](int which) { return bars_u32 + uint32_t(which) * 8; };
    // False when the wait ran out here or somewhere else in the CTA (lanes may disagree on that); raises the flag that ends the others.
    auto wait = [&](int which, uint32_t parity) {
        const bool ok = wait_or_abort(bar(which), parity & 1u, s_abort, kShortWaits ? p.wait_limit : kMbarWaitLimit);
        if (!ok) {
            *s_abort = 1;
        }
        return ok;
    };
    // For what is on its way in any case: not cut short by another warp's failure.
    auto drain = [&](int which, uint32_t parity) {
        if (!mbar_wait_bounded(bar(which), parity & 1u, kMbarWaitLimit)) {
            *s_abort = 1;
        }
        __syncwarp();
    };
    // A warp's place on the line waits in shared memory while its blocks run: a register that is spilled there is fetched from L2 (the
    // operands leave no L1), and a dozen such loads per block cost as much as the block.
    Place *place = reinterpret_cast<Place *>(s_sched + kSchedInts + warp * kPlaceInts);
    auto keep_place = [&](const Walker &w, const Fragment &f, int pos) {
        __syncwarp();
        if (lane == 0) {
            place->w = w;
            place->f = f;
            place->pos = pos;
        }
        __syncwarp();
    };
    keep_place(walker, Fragment{}, piece_begin);
    // The next fragment of the piece, in this warp's place.
    auto next_fragment = [&](Walker &w, Fragment &f) {
        int pos = place->pos;
        w = place->w;
        const bool found = locate(p, w, pos, s_line[1], f);
        keep_place(w, f, pos + (found ? f.units : 0));
        return found;
    };

    // (setmaxnreg inside each branch: where they met again the compiler would keep to the smaller count)
    if (warp >= kProducerWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kOtherRegs));
        if (warp == kProducerWarp) {
            // ================================ producer: TMA tiles of K and V =========================================
            bool alive = true;
            int stage = 0;
            uint32_t turn = 0; // times the ring has been filled
            while (alive) {
                Fragment f;
                Walker w;
                if (!next_fragment(w, f)) {
                    break;
                }
                const int n = f.b1 - f.b0, kept_blocks = w.g.kept_blocks;
                const int n_pages = (tile_kv_hi(w.g, f.qb) + kPage - 1) / kPage;
                const int seq_row = (!p.contiguous && p.seq_ids) ? p.seq_ids[f.a] : f.a;
                const long long tbase = (long long)seq_row * p.table_stride;
                // Page numbers come 4 blocks (32 table entries) at a time, and the group after the current one is requested a group early.
                // Behind a tile's last page its last page comes again: hidden keys have weight 0, and what they are multiplied by is then
                // always a row of this sequence.
                auto load_group = [&](int blk0) {
                    const int b = blk0 + lane / kPagesPerBlock;
                    const int idx = min((kWin && b >= kept_blocks ? b + f.gap : b) * kPagesPerBlock + lane % kPagesPerBlock, n_pages - 1);
                    return p.contiguous ? idx : p.block_table[tbase + idx]; // block b of a tensor is its tokens [128 b, 128 b + 128)
                };
                constexpr int kGroup = 32 / kPagesPerBlock;
                int group = load_group(f.b0), next_group = load_group(f.b0 + kGroup);
                for (int i = 0; i < n && alive; ++i) {
                    if (i > 0 && i % kGroup == 0) {
                        group = next_group;
                        next_group = load_group(f.b0 + i + kGroup);
                    }
                    int page = __shfl_sync(0xffffffffu, group, i % kGroup * kPagesPerBlock + lane % kPagesPerBlock);
                    if (!p.contiguous && (page < 0 || page >= p.num_pages)) {
                        atomicOr(p.error_flag, kErrBadPage);
                        page = 0;
                    }
                    const int row = int((p.page0 + page) * 2); // K of the page; V is the next index
#pragma unroll
                    for (int is_v = 0; is_v < 2; ++is_v) {
                        if (turn > 0 && !__all_sync(0xffffffffu, wait(kBarEmpty + stage, turn - 1))) {
                            alive = false;
                            break;
                        }
                        const uint32_t full = bar(kBarFull + stage), at = ring_u32 + stage * kStageBytes;
                        if (lane == 0) {
                            mbar_arrive_expect_tx(full, kStageBytes);
                        }
                        __syncwarp();
                        if (is_v && lane < kPagesPerBlock) {
                            // V: ONE box per page -- 64 dims x 16 tokens x the 2 halves of the row -- lands as [half][16 tokens][128 B], which is
                            // what the MN-major B operand of P.V reads 16 keys at a time
                            if (p.contiguous) {
                                tma_load_4d(at + lane * 4096, &tmap_v, 0, page * kPage, 0, f.kvh, full);
                            } else {
                                tma_load_5d(at + lane * 4096, &tmap_v, 0, 0, 0, f.kvh, row + 1, full);
                            }
                        } else if (!is_v && lane < 2 * kPagesPerBlock) {
                            // K: the K-major B operand of Q.K^T wants the keys of a block side by side in each 64-dim half, so a page is two
                            // boxes of 64 dims x 16 tokens
                            const int half = lane / kPagesPerBlock;
                            const uint32_t to = at + half * kPieceBytes + lane % kPagesPerBlock * 2048;
                            if (p.contiguous) {
                                tma_load_3d(to, &tmap, half * 64, f.kvh, page * kPage, full); // (tokens past the end read as 0)
                            } else {
                                tma_load_4d(to, &tmap, half * 64, 0, f.kvh, row, full);
                            }
                        }
                        if (++stage == kStages) {
                            stage = 0;
                            ++turn;
                        }
                    }
                }
            }
            for (int load = max(int(turn) * kStages + stage - kStages, 0); load < int(turn) * kStages + stage; ++load) {
                drain(kBarFull + load % kStages, uint32_t(load / kStages));
            }
        } else if (warp <= kMmaWarp + 1) {
            // ================================ MMA issuers, one warp per half ========================================
            // tcgen05.mma is accepted at the pace of the tensor pipe, a few instructions ahead: with one warp for both halves the pipe stood idle
            // through every wait, commit and loop step between batches (2100 of a block's 4200 clocks). With two, one half's batch runs under the
            // other's waits. The whole warp walks the blocks and one lane issues: descriptors then come from uniform registers.
            // A lane whose wait ran out issues nothing any more and skips its later waits, but walks on: the warp stays together without a vote per
            // wait (with one, a prompt of 8192 took 587 instead of 558 us).
            const int h = __shfl_sync(0xffffffffu, warp, 0) - kMmaWarp;
            constexpr uint32_t idesc_qk = make_idesc(kBf16, false, kHalf, kKeys), idesc_pv = make_idesc(kBf16, true, kHalf, kD);
            const uint32_t tmem_s = __shfl_sync(0xffffffffu, tmem_base, 0) + kColS + h * kKeys, tmem_o = __shfl_sync(0xffffffffu, tmem_base, 0) + kColO + h * kD;
            const uint64_t q_desc = smem_desc_sw128(base_u32 + h * kQBytes, 0, 1024), k_desc = smem_desc_sw128(ring_u32, 0, 1024),
                           v_desc = smem_desc_sw128(ring_u32, 2048, 1024);
            const bool leader = elect_one();
            bool ok = true;
            int stage = 0;
            uint32_t turn = 0, p_turn = 0, q_turn = 0, my_turn = 0;
            // Where both halves have rows their batches alternate: left to themselves they fall into step, both softmaxes at once (and short of
            // exponentials), then both halves' MMAs (3600 clocks a block against 3050).
            bool two = false;
            auto take_turn = [&]() {
                if (two && (h == 1 || my_turn > 0)) {
                    ok = ok && wait(kBarTurn + h, h == 1 ? my_turn : my_turn - 1);
                }
                my_turn += two ? 1u : 0u;
            };
            auto take_stage = [&]() { // the next stage of the ring, once it has landed
                const int s = stage;
                ok = ok && wait(kBarFull + s, turn);
                stage = s + 1 == kStages ? 0 : s + 1;
                turn += s + 1 == kStages ? 1u : 0u;
                return s;
            };
            auto issue_qk = [&](int s) {
                const uint64_t k = k_desc + uint64_t(s * (kStageBytes >> 4));
                if (leader && ok) {
#pragma unroll
                    for (int ks = 0; ks < kD / 16; ++ks) {
                        umma_f16(tmem_s, q_desc + uint64_t(((ks >> 2) * kQPiece + (ks & 3) * 32) >> 4), k + uint64_t(((ks >> 2) * kPieceBytes + (ks & 3) * 32) >> 4),
                                 idesc_qk, ks > 0 ? 1u : 0u);
                    }
                }
            };
            auto commit = [&](int which) {
                if (leader && ok) {
                    umma_commit(bar(which));
                    if (two) {
                        mbar_arrive(bar(kBarTurn + 1 - h));
                    }
                }
                __syncwarp();
            };
            for (;;) {
                Fragment f;
                {
                    Walker w;
                    if (!next_fragment(w, f)) {
                        break;
                    }
                }
                const int n = __shfl_sync(0xffffffffu, f.b1 - f.b0, 0);
                two = __shfl_sync(0xffffffffu, f.rows, 0) > kHalf;
                if (h == 1 && !two) { // no rows: see the stages pass (every phase in order) and free them
                    for (int i = 0; i < 2 * n; ++i) {
                        const int s = take_stage();
                        if (ok && lane == 0) {
                            mbar_arrive(bar(kBarEmpty + s));
                        }
                    }
                    continue;
                }
                const int k0 = take_stage();
                ok = ok && wait(kBarQ + h, q_turn++);
                take_turn();
                issue_qk(k0);
                commit(kBarS + h);
                for (int i = 0; i < n; ++i) {
                    const bool more = i + 1 < n;
                    const int v_at = take_stage(), k_at = more ? take_stage() : 0;
                    const uint64_t v = v_desc + uint64_t(v_at * (kStageBytes >> 4));
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        ok = ok && wait(kBarP + h * 2 + part, p_turn);
                        if (part == 0) {
                            take_turn();
                        }
                        tc_fence_after();
                        if (leader && ok) {
#pragma unroll
                            for (int k4 = 0; k4 < kPagesPerBlock / 2; ++k4) {
                                // B = 16 keys (one page) x 128 dims of V, MN-major: 8-key groups 1 KiB apart, the page's two 64-dim halves 2 KiB
                                // apart, pages 4 KiB apart. A = P rows x 16 keys from tensor memory: 8 columns of packed pairs per step
                                const int kk = part * (kPagesPerBlock / 2) + k4;
                                umma_f16_ts(tmem_o, tmem_s + kk * 8, v + uint64_t(kk * 4096 >> 4), idesc_pv, i > 0 || kk > 0 ? 1u : 0u);
                            }
                        }
                    }
                    ++p_turn;
                    if (more) {
                        issue_qk(k_at);
                    }
                    commit((more ? kBarS : kBarO) + h);
                }
            }
            if (leader) {
                umma_commit(bar(kBarDrain + h));
            }
            __syncwarp();
            drain(kBarDrain + h, 0);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kSoftmaxRegs));
        // ================================ softmax: one row per thread ===========================================
        const int h = warp >> 2, row = tid & (kHalf - 1); // half of the tile, TMEM lane
        const uint32_t lane_base = tmem_base + (uint32_t((warp & 3) * 32) << 16);
        const uint32_t tmem_s = lane_base + kColS + h * kKeys, tmem_o = lane_base + kColO + h * kD;
        const uint32_t q_u32 = base_u32 + h * kQBytes;
        auto per_group = [&](int x) { return p.group == 1 ? x : int(__umulhi(uint32_t(x), p.group_inverse)); };
        // Q rows of this half, 16 bytes per store, into the K-major 128-byte-swizzled layout; rows past the chunk are zero. All loads first,
        // then all stores: the stores are volatile asm, which no load may pass.
        auto load_q = [&](const Fragment &f, const SeqGeom &g) {
            constexpr int kIter = kHalf * 16 / kSoftmaxThreads;
            uint4 vals[kIter];
#pragma unroll
            for (int it = 0; it < kIter; ++it) {
                const int r = (row >> 4) + it * (kSoftmaxThreads / 16), cc = row & 15, x = f.qb * kRows + h * kHalf + r, t = per_group(x);
                vals[it] = make_uint4(0u, 0u, 0u, 0u);
                if (t < g.q_len) {
                    vals[it] = *reinterpret_cast<const uint4 *>(static_cast<const char *>(p.q) + cc * 16 +
                                                                ((long long)(g.q_start + t) * p.nh + f.kvh * p.group + (x - t * p.group)) * (kD * 2));
                }
            }
#pragma unroll
            for (int it = 0; it < kIter; ++it) {
                const int r = (row >> 4) + it * (kSoftmaxThreads / 16), cc = row & 15;
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(q_u32 + (cc >> 3) * kQPiece + r * 128 + (((cc & 7) ^ (r & 7)) << 4)),
                             "r"(vals[it].x), "r"(vals[it].y), "r"(vals[it].z), "r"(vals[it].w)
                             : "memory");
            }
            fence_proxy_async_smem(); // read by the async proxy
            mbar_arrive(bar(kBarQ + h));
        };
        // A lane whose wait ran out goes on with what it finds, so that the warp stays together (without a vote per block, which took 2 % of
        // a prompt, and with one flag less in the block loop) and the named barrier and the arrival counts below see all 128 threads every
        // time. Nothing of a fragment is stored once the CTA has given up.
        uint32_t s_turn = 0, o_turn = 0;
        // stages that this half has seen read: K of block b is load 2 b of the CTA, V load 2 b + 1
        int done = 0; // blocks of earlier fragments
        auto free_stage = [&](int load) {
            if (row == 0) {
                mbar_arrive(bar(kBarEmpty + load % kStages));
            }
        };
        bool more = false;
        auto move_on = [&]() { // to the next fragment that has rows for this half: Q rows loaded
            Walker w;
            Fragment f;
            while ((more = next_fragment(w, f)) && h == 1 && f.rows <= kHalf) {
                done += f.b1 - f.b0;
            }
            if (more) {
                load_q(f, w.g);
            }
        };
        move_on();
        while (more) {
            Fragment f = place->f;
            SeqGeom g = place->w.g;
            const int n = f.b1 - f.b0;
            const int x = f.qb * kRows + h * kHalf + row, t = per_group(x), head = f.kvh * p.group + (x - t * p.group);
            const int last_visible = t + g.off; // keys j <= last_visible (and < kv_len) take part
            const int n_seen = min(last_visible + 1, g.kv_len);
            float m_used = -INFINITY, l = 0.f;
            const float fade_a = kFade ? p.fade_a[head] : 0.f, fade_b = kFade ? p.fade_b[head] : 0.f;
            for (int i = 0; i < n; ++i) {
                wait(kBarS + h, s_turn++);
                tc_fence_after();
                free_stage(2 * (done + i));
                if (i >= 1) {
                    free_stage(2 * (done + i) - 1);
                }
                const int j0 = (f.b0 + i + (kWin && f.b0 + i >= g.kept_blocks ? f.gap : 0)) * kKeys;
                const int n_ok = min(n_seen - j0, kKeys);                     // visible columns are [0, n_ok)
                const int n_lo = kWin ? last_visible - p.window + 1 - j0 : 0; // columns below n_lo lie before the row's window,
                const int n_kept = kWin ? p.keep_first - j0 : 0;              // those below n_kept are seen all the same
                uint32_t sr[kKeys / 32][32];
#pragma unroll
                for (int c = 0; c < kKeys / 32; ++c) {
                    tmem_ld32_nowait(tmem_s + c * 32, sr[c]);
                }
                tmem_wait_ld();
                float to_log2 = p.scale_log2; // what the scores still have to be multiplied by
                if constexpr (kFade) {
                    // (distances are exact; those of hidden keys may be negative, whatever comes of them is masked below)
                    const float d0 = float(last_visible - j0);
#pragma unroll
                    for (int c = 0; c < kKeys / 32; ++c) {
#pragma unroll
                        for (int k = 0; k < 32; k += 2) {
                            float a0, a1, x0, x1;
                            fma2(a0, a1, d0 - float(c * 32 + k), d0 - float(c * 32 + k + 1), fade_b, 1.f);
                            fma2(x0, x1, __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 1]), p.scale_log2, 0.f);
                            sr[c][k] = __float_as_uint(fmaf(-fade_a, fast_log2(a0), x0));
                            sr[c][k + 1] = __float_as_uint(fmaf(-fade_a, fast_log2(a1), x1));
                        }
                    }
                    to_log2 = 1.f;
                } else if (!(p.scale_log2 > 0.f)) { // a scale that is not positive does not keep the order of the scores
#pragma unroll
                    for (int c = 0; c < kKeys / 32; ++c) {
#pragma unroll
                        for (int k = 0; k < 32; ++k) {
                            sr[c][k] = __float_as_uint(__uint_as_float(sr[c][k]) * p.scale_log2);
                        }
                    }
                    to_log2 = 1.f;
                }
                // Most blocks lie wholly below the diagonal: the whole warp then skips the mask (warp-uniform choice), and otherwise the 32-column
                // pieces that every row of the warp sees. Hidden scores become -inf: 2^(-inf * scale - m) = 0.
                if (!__all_sync(0xffffffffu, n_ok >= kKeys && (!kWin || n_lo <= 0 || n_kept >= kKeys))) {
                    auto below = [](int n) { return n <= 0 ? 0u : 0xffffffffu >> (32 - min(n, 32)); }; // bits 0 .. n - 1
#pragma unroll
                    for (int c = 0; c < kKeys / 32; ++c) {
                        uint32_t seen = below(n_ok - c * 32);
                        if constexpr (kWin) {
                            seen &= ~below(n_lo - c * 32) | below(n_kept - c * 32);
                        }
                        if (!__all_sync(0xffffffffu, seen == 0xffffffffu)) {
#pragma unroll
                            for (int k = 0; k < 32; ++k) {
                                sr[c][k] = (seen >> k) & 1u ? sr[c][k] : 0xff800000u;
                            }
                        }
                    }
                }
                // row maximum as eight independent chains
                float mx8[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    mx8[u] = -INFINITY;
                }
#pragma unroll
                for (int c = 0; c < kKeys / 32; ++c) {
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        mx8[k & 7] = max3(mx8[k & 7], __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 16]));
                    }
                }
                const float mx = max3(max3(mx8[0], mx8[1], mx8[2]), max3(mx8[3], mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7])) * to_log2;
                // The running max only moves when it grew by more than 2^8: P and the row sum both use m_used, so the result is exact
                // either way, and O is rescaled rarely. (The scores' arrival says that the product of the block before is done.)
                float alpha = 1.f;
                const bool grow = mx > m_used + kRescaleThreshold;
                if (grow) {
                    alpha = fast_exp2(m_used - mx); // 0 on the fragment's first visible block
                    m_used = mx;
                }
                l *= alpha;
                if (i >= 1 && __any_sync(0xffffffffu, grow)) { // (the first product of a fragment overwrites O)
#pragma unroll
                    for (int c = 0; c < kD / 32; ++c) {
                        float v[32];
                        tmem_ld32(tmem_o + c * 32, v);
#pragma unroll
                        for (int k = 0; k < 32; ++k) {
                            v[k] *= alpha;
                        }
                        tmem_st32(tmem_o + c * 32, v);
                    }
                }
                const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
                float l0 = 0.f, l1 = 0.f, l2 = 0.f, l3 = 0.f; // independent sums: short dependency chains
#pragma unroll
                for (int c = 0; c < kKeys / 32; ++c) { // 32 keys = 16 columns of packed pairs over the scores
                    float packed[16];
#pragma unroll
                    for (int k = 0; k < 32; k += 2) {
                        float x0, x1;
                        fma2(x0, x1, __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 1]), to_log2, neg_m);
                        const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
                        // With a distance penalty a few near keys dominate a row: there the sum is of the weights as they are multiplied, rounded
                        // to 16 bits, and the row is off by the rounding of its result alone. (Everywhere it would cost 9 % of a long prompt.)
                        const uint32_t w = pack2<kBf16>(p0, p1);
                        const float2 r = kFade ? unpack2<kBf16>(w) : make_float2(p0, p1);
                        if (k & 2) {
                            add2(l2, l3, r.x, r.y);
                        } else {
                            add2(l0, l1, r.x, r.y);
                        }
                        packed[k >> 1] = __uint_as_float(w);
                    }
                    tmem_st16(tmem_s + c * 16, packed);
                    if (c & 1) {
                        tmem_wait_st();
                        tc_fence_before();
                        mbar_arrive(bar(kBarP + h * 2 + (c >> 1)));
                    }
                }
                l += (l0 + l1) + (l2 + l3);
            }
            // ---- Q rows of the next fragment: every Q K^T of this one has finished (its last scores were read above) ----------
            asm volatile("" ::: "memory");
            f = place->f;
            g = place->w.g;
            const int last_load = 2 * (done + n) - 1; // V of the last block
            done += n;
            move_on();
            // ---- epilogue of the fragment ---------------------------------------------------------------------------
            wait(kBarO + h, o_turn++);
            tc_fence_after();
            free_stage(last_load);
            const bool dead = __any_sync(0xffffffffu, *s_abort != 0) != 0;
            const bool whole = f.b0 == 0 && f.b1 == f.tile_nblk;
            bool store_rows = whole;
            float w_own = 1.f, l_all = l, m_all = m_used;
            const int piece = s_line[0], first_slot = f.tile_begin / piece, last_slot = (f.tile_begin + f.tile_nblk - 1) / piece;
            auto part_of = [&](int s2) { // a fragment's place in the workspace: 1 for the one that begins its tile (and goes on in the next CTA)
                return p.partials + ((long long)(s2 * 2 + (s2 * piece <= f.tile_begin ? 1 : 0)) * 2 + h) * kPartialFloats;
            };
            if (!whole) {
                float *part = p.partials + ((long long)(slot * 2 + (f.b0 == 0 ? 1 : 0)) * 2 + h) * kPartialFloats;
                if (!dead) {
#pragma unroll
                    for (int c4 = 0; c4 < 4; ++c4) {
                        float v[32];
                        tmem_ld32(tmem_o + c4 * 32, v);
#pragma unroll
                        for (int q8 = 0; q8 < 8; ++q8) {
                            reinterpret_cast<float4 *>(part)[(c4 * 8 + q8) * kHalf + row] = make_float4(v[q8 * 4], v[q8 * 4 + 1], v[q8 * 4 + 2], v[q8 * 4 + 3]);
                        }
                    }
                    part[kHalf * kD + row] = m_used;
                    part[kHalf * kD + kHalf + row] = l;
                }
                named_barrier_sync(1 + h, kSoftmaxThreads);
                if (row == 0) { // (one release for all of the half's stores: the barrier made them this thread's to publish)
                    int before;
                    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;\n" : "=r"(before) : "l"(p.counters + first_slot * 2 + h) : "memory");
                    const bool last = before == last_slot - first_slot;
                    if (last) {
                        p.counters[first_slot * 2 + h] = 0; // ready for the next launch
                    }
                    s_sched[3 * kWarps + 2 + h] = last ? 1 : 0;
                }
                named_barrier_sync(1 + h, kSoftmaxThreads);
                store_rows = s_sched[3 * kWarps + 2 + h] != 0;
                if (store_rows && !dead) {
                    // weights 2^(m_i - m); sums run over the fragments in the order of their CTAs, this one's terms in its place: the
                    // result does not depend on which fragment happened to arrive last
                    for (int s2 = first_slot; s2 <= last_slot; ++s2) {
                        if (s2 != slot) {
                            m_all = fmaxf(m_all, __ldcg(part_of(s2) + kHalf * kD + row));
                        }
                    }
                    w_own = m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_all);
                    l_all = 0.f;
                    for (int s2 = first_slot; s2 <= last_slot; ++s2) {
                        const float m2 = s2 == slot ? m_used : __ldcg(part_of(s2) + kHalf * kD + row);
                        const float l2 = s2 == slot ? l : __ldcg(part_of(s2) + kHalf * kD + kHalf + row);
                        l_all = fmaf(l2, m2 == -INFINITY ? 0.f : fast_exp2(m2 - m_all), l_all);
                    }
                }
            }
            if (store_rows && !dead) {
                float inv = l_all > 0.f ? 1.f / l_all : 0.f;
                if (kWin && p.row_scale != nullptr && t < g.q_len) {
                    inv *= p.row_scale[(long long)(g.q_start + t) * p.nh + head];
                }
                char *out_row = static_cast<char *>(p.out) + ((long long)(g.q_start + t) * p.out_stride + head * kD) * 2;
#pragma unroll
                for (int c2 = 0; c2 < 2; ++c2) { // 64 columns at a time
                    float v[64];
                    auto own = [&](bool first, float w) { // this fragment's columns
                        float o[32];
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            tmem_ld32(tmem_o + c2 * 64 + c * 32, o);
#pragma unroll
                            for (int k = 0; k < 32; ++k) {
                                v[c * 32 + k] = first ? o[k] : fmaf(o[k], w, v[c * 32 + k]);
                            }
                        }
                    };
                    if (whole) {
                        own(true, 1.f);
                    } else {
#pragma unroll
                        for (int k = 0; k < 64; ++k) {
                            v[k] = 0.f;
                        }
                        for (int s2 = first_slot; s2 <= last_slot; ++s2) {
                            if (s2 == slot) {
                                own(false, w_own);
                                continue;
                            }
                            const float *other = part_of(s2);
                            const float m2 = __ldcg(other + kHalf * kD + row);
                            const float w2 = m2 == -INFINITY ? 0.f : fast_exp2(m2 - m_all);
#pragma unroll
                            for (int q16 = 0; q16 < 16; ++q16) {
                                const float4 o = __ldcg(reinterpret_cast<const float4 *>(other) + (c2 * 16 + q16) * kHalf + row);
                                v[q16 * 4] = fmaf(o.x, w2, v[q16 * 4]);
                                v[q16 * 4 + 1] = fmaf(o.y, w2, v[q16 * 4 + 1]);
                                v[q16 * 4 + 2] = fmaf(o.z, w2, v[q16 * 4 + 2]);
                                v[q16 * 4 + 3] = fmaf(o.w, w2, v[q16 * 4 + 3]);
                            }
                        }
                    }
                    if (t < g.q_len && p.out_wide) {
                        // a thread owns a row: a 16-byte store fills half a 32-byte sector and the other half comes with the next
                        // instruction; 32-byte stores halve the write transactions of the epilogue
#pragma unroll
                        for (int q4 = 0; q4 < 4; ++q4) {
                            uint32_t w[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                w[e] = pack2<kBf16>(v[q4 * 16 + 2 * e] * inv, v[q4 * 16 + 2 * e + 1] * inv);
                            }
                            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(out_row + c2 * 128 + q4 * 32),
                                         "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                                         : "memory");
                        }
                    } else if (t < g.q_len) {
#pragma unroll
                        for (int q8 = 0; q8 < 8; ++q8) {
                            uint4 w;
                            w.x = pack2<kBf16>(v[q8 * 8 + 0] * inv, v[q8 * 8 + 1] * inv);
                            w.y = pack2<kBf16>(v[q8 * 8 + 2] * inv, v[q8 * 8 + 3] * inv);
                            w.z = pack2<kBf16>(v[q8 * 8 + 4] * inv, v[q8 * 8 + 5] * inv);
                            w.w = pack2<kBf16>(v[q8 * 8 + 6] * inv, v[q8 * 8 + 7] * inv);
                            *reinterpret_cast<uint4 *>(out_row + c2 * 128 + q8 * 16) = w;
                        }
                    }
                }
            }
            tc_fence_before(); // the O reads above come before the next fragment's P arrival in program order
        }
    }

    // ---- teardown: everyone is done with TMEM before the allocating warp frees it ----------------------------------
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *s_abort != 0) {
        atomicOr(p.error_flag, kErrTimeout);
    }
    if (warp == kMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

} // namespace

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn chunk_encode_fn() {
    static EncodeTiledFn fn = [] {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &res) != cudaSuccess ||
            res != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            return EncodeTiledFn(nullptr);
        }
        return reinterpret_cast<EncodeTiledFn>(sym);
    }();
    return fn;
}

// CTAs of the fixed grid: one per SM
int chunk_slots() {
    static int slots[64] = {};
    int dev = 0;
    LLAISYS_CUDA_CHECK(cudaGetDevice(&dev));
    int &n = slots[dev & 63];
    if (n == 0) {
        int sms = 0;
        LLAISYS_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        n = sms > 0 ? sms : 1;
    }
    return n;
}

template <bool kBf16, int kForm, bool kShortWaits = false>
void launch(cudaStream_t s, const CUtensorMap &tmap, const CUtensorMap &tmap_v, const ChunkParams &p, int grid, bool overlap) {
    static std::once_flag once[64];
    int dev = 0;
    LLAISYS_CUDA_CHECK(cudaGetDevice(&dev));
    std::call_once(once[dev & 63], [] {
        LLAISYS_CUDA_CHECK(cudaFuncSetAttribute(paged_prefill_tc_kernel<kBf16, kForm, kShortWaits>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBytes)));
    });
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(unsigned(kThreads));
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    LLAISYS_CUDA_CHECK(cudaLaunchKernelEx(&cfg, paged_prefill_tc_kernel<kBf16, kForm, kShortWaits>, tmap, tmap_v, p));
}

} // namespace

void attention_prefill_tc_scratch(size_t *floats, size_t *counters) {
    const size_t slots = size_t(chunk_slots()); // (two halves of two fragments per CTA; attention_narrow_tc.cu needs no more)
    *floats = 4 * slots * size_t(kPartialFloats);
    *counters = 2 * slots;
}

int make_kv_tile_tensor_map(void *out_256_bytes, void *pool_base, uint64_t total_rows, uint32_t nkvh,
                            llaisysDataType_t dtype) {
    if (dtype != LLAISYS_DTYPE_BF16 && dtype != LLAISYS_DTYPE_F16) {
        return -1;
    }
    if (total_rows == 0 || nkvh == 0 || total_rows % (uint64_t(kPage) * nkvh) != 0 || total_rows >= (uint64_t(1) << 31) ||
        reinterpret_cast<uintptr_t>(pool_base) % 16 != 0) {
        return -1;
    }
    EncodeTiledFn encode = chunk_encode_fn();
    if (encode == nullptr) {
        return -1;
    }
    // Same 4-D view of the pool as the decode kernel's map -- [page-and-K|V][kv-head][slot][128 elements] -- with a
    // box of one half-tile: 64 elements x 16 slots (2 KiB, 128-byte swizzle).
    const cuuint64_t dims[4] = {cuuint64_t(kD), cuuint64_t(kPage), cuuint64_t(nkvh), cuuint64_t(total_rows / (kPage * nkvh))};
    const cuuint64_t strides[3] = {cuuint64_t(kD * 2), cuuint64_t(kPage * kD * 2), cuuint64_t(kPage * kD * 2) * nkvh};
    const cuuint32_t box[4] = {64, cuuint32_t(kPage), 1, 1};
    const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
    CUtensorMap map;
    const CUresult rc =
        encode(&map, dtype == LLAISYS_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
               pool_base, dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) {
        return -1;
    }
    // The second map is for V: a 5-D view [page-and-K|V][kv-head][half of the row][slot][64 elements] whose box is a whole
    // tile as two 64-dim halves, 64 x 16 x 2 (4 KiB): one copy per page instead of two.
    const cuuint64_t dims5[5] = {64, cuuint64_t(kPage), 2, cuuint64_t(nkvh), cuuint64_t(total_rows / (kPage * nkvh))};
    const cuuint64_t strides5[4] = {cuuint64_t(kD * 2), 128, cuuint64_t(kPage * kD * 2), cuuint64_t(kPage * kD * 2) * nkvh};
    const cuuint32_t box5[5] = {64, cuuint32_t(kPage), 2, 1, 1};
    const cuuint32_t elem_strides5[5] = {1, 1, 1, 1, 1};
    CUtensorMap map_v;
    const CUresult rc_v =
        encode(&map_v, dtype == LLAISYS_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5,
               pool_base, dims5, strides5, box5, elem_strides5, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc_v != CUDA_SUCCESS) {
        return -1;
    }
    static_assert(sizeof(CUtensorMap) == 128, "two maps in 256 bytes");
    memcpy(out_256_bytes, &map, sizeof(map));
    memcpy(static_cast<unsigned char *>(out_256_bytes) + sizeof(map), &map_v, sizeof(map_v));
    return 0;
}

namespace {

// [tokens][nkvh][128] 16-bit tensor -> 3-D map (dims 128, nkvh, tokens) with a box of 64 dims x 1 head x 16 tokens: the
// tile lands in shared memory exactly like a page-pool tile; rows past the last token are out of bounds and read as 0.
bool contiguous_kv_map(CUtensorMap *out, const void *base, const KVView &kv, uint64_t tokens, bool bf16) {
    EncodeTiledFn encode = chunk_encode_fn();
    if (encode == nullptr || tokens == 0 || tokens >= (uint64_t(1) << 31)) {
        return false;
    }
    const cuuint64_t dims[3] = {cuuint64_t(kD), cuuint64_t(kv.nkvh), cuuint64_t(tokens)};
    const cuuint64_t strides[2] = {cuuint64_t(kv.head_stride) * 2, cuuint64_t(kv.token_stride) * 2};
    const cuuint32_t box[3] = {64, 1, cuuint32_t(kPage)};
    const cuuint32_t elem_strides[3] = {1, 1, 1};
    return encode(out, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base),
                  dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same tensor for V: 4-D (64 dims, tokens, half of the row, kv-head) with a box of 64 x 16 x 2 x 1, one copy per 16 tokens.
bool contiguous_v_map(CUtensorMap *out, const void *base, const KVView &kv, uint64_t tokens, bool bf16) {
    EncodeTiledFn encode = chunk_encode_fn();
    if (encode == nullptr || tokens == 0 || tokens >= (uint64_t(1) << 31)) {
        return false;
    }
    const cuuint64_t dims[4] = {64, cuuint64_t(tokens), 2, cuuint64_t(kv.nkvh)};
    const cuuint64_t strides[3] = {cuuint64_t(kv.token_stride) * 2, 128, cuuint64_t(kv.head_stride) * 2};
    const cuuint32_t box[4] = {64, cuuint32_t(kPage), 2, 1};
    const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
    return encode(out, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(base),
                  dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

} // namespace

namespace {

// Calls that take less time in tiles of 128 rows of ONE head, two CTAs per SM, blocks of 64 keys (attention_narrow_tc) than in 256 packed
// rows. Times of both, narrow first.
bool narrow(const AttnBatch &batch, int nkvh, int sms, bool paged) {
    const int64_t heads = int64_t(batch.n_seqs) * batch.nh, tiles = heads * ((batch.max_q_len + 127) / 128);
    const int64_t keys = batch.window > 0 ? std::min<int64_t>(batch.max_kv_len, int64_t(batch.window) + batch.keep_first + batch.max_q_len)
                                          : batch.max_kv_len;
    // One block of 64 keys and one tile per SM at most: half of a block here would be padding (64 tokens, 32 / 8 heads, 11.2 and 15.1 us; 128
    // tokens are 17.5 and 15.3).
    if (keys <= 64 && tiles <= sms) {
        return true;
    }
    // A head per kv head and up to 128 queries: a tile here fills one half and the SM's other softmax group idles. With more tiles than SMs
    // that shows (64 chunks of 64 behind 1000, 16 / 16 heads, two layers: 271 and 301; of 64 behind nothing 94 and 122); not between, where
    // whole tiles of few blocks still win (24 chunks of 32 behind 200, 8 / 8 heads: 60 and 46), unless the waves are many and full.
    if (batch.nh == nkvh && batch.total_q <= 128 * int64_t(batch.n_seqs) && heads > sms) {
        return keys <= 64 || keys > 768 || (batch.total_q >= 64 * int64_t(batch.n_seqs) && heads > 2 * int64_t(sms));
    }
    // Plain tensors, with no kernel in front whose end hides this kernel's start, and few tiles to spread over the chip: 512 queries x 1000
    // keys, 12 / 2 heads, 25.5 and 27.8; 256 x 3000 32.9 and 35.5 (x 600 23.6 and 21.8, x 8000 54 and 48, 1024 x 3000 41 and 39.7).
    return !paged && batch.nh > nkvh && keys > 640 && keys <= 4096 && tiles <= 48;
}

} // namespace

int attention_prefill_tc(stream_t stream, llaisysDataType_t dtype, const KVView &kv, const AttnBatch &batch,
                         const void *q, float scale, const AttnOut &out, const AttnScratch &scratch) {
    int32_t *error_flag = scratch.error_flag;
    const bool bf16 = dtype == LLAISYS_DTYPE_BF16;
    if (!(bf16 || dtype == LLAISYS_DTYPE_F16) || kv.d != kD || kv.page_size != kPage || kv.nkvh <= 0 || out.out == nullptr ||
        out.part != nullptr || batch.nh % kv.nkvh != 0 || batch.n_seqs <= 0 || batch.max_q_len <= 0 || error_flag == nullptr ||
        reinterpret_cast<uintptr_t>(q) % 16 != 0 || reinterpret_cast<uintptr_t>(out.out) % 16 != 0) {
        return -1;
    }
    // Two kinds of K/V: a page pool with a block table (one tensor map over the pool, made with the cache), or the
    // legacy operator's plain [tokens, nkvh, 128] tensors of one sequence (two maps made here).
    const bool paged = kv.block_table != nullptr;
    if (paged && (kv.tma_tile_desc == nullptr || batch.kv_lens == nullptr || batch.q_starts == nullptr)) {
        return -1;
    }
    const bool contiguous = !paged && batch.n_seqs == 1 && batch.q_starts == nullptr && batch.kv_lens == nullptr &&
                            batch.seq_ids == nullptr && batch.const_q_len > 1 && batch.const_kv_len >= batch.const_q_len &&
                            kv.head_stride == kD && kv.token_stride == int64_t(kv.nkvh) * kD &&
                            reinterpret_cast<uintptr_t>(kv.k_base) % 16 == 0 && reinterpret_cast<uintptr_t>(kv.v_base) % 16 == 0;
    if (!paged && !contiguous) {
        return -1;
    }
    ChunkParams p{};
    p.page0 = paged ? kv.tma_page0 : 0;
    p.block_table = kv.block_table;
    p.table_stride = kv.table_stride;
    p.num_pages = kv.num_pages;
    p.seq_ids = batch.seq_ids;
    p.kv_lens = batch.kv_lens;
    p.q_starts = batch.q_starts;
    p.contiguous = contiguous ? 1 : 0;
    p.const_q_len = batch.const_q_len;
    p.const_kv_len = batch.const_kv_len;
    p.n_seqs = batch.n_seqs;
    p.nkvh = kv.nkvh;
    p.group = batch.nh / kv.nkvh;
    p.nh = batch.nh;
    p.group_inverse = uint32_t(((uint64_t(1) << 32) + uint64_t(p.group) - 1) / uint64_t(p.group));
    p.q = q;
    p.out = out.out;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.error_flag = error_flag;
    p.wait_limit = kv.wait_limit;
    // the workspace of the split tiles: the halves of two fragments per CTA, and an arrival counter per half
    const int grid = chunk_slots();
    if (scratch.partials == nullptr || scratch.counters == nullptr ||
        scratch.partials_floats < 4 * size_t(grid) * size_t(kPartialFloats) || scratch.counters_len < 2 * size_t(grid) ||
        reinterpret_cast<uintptr_t>(scratch.partials) % 16 != 0) {
        return -1;
    }
    const bool fading = batch.fade_a != nullptr, windowed = batch.window > 0 || out.row_scale != nullptr || out.row_stride != 0 || fading;
    if ((windowed && !paged) || out.row_stride % 8 != 0) {
        return -1;
    }
    p.window = windowed && batch.window <= 0 ? kv.table_stride * kPage : batch.window; // (a factor alone: a window nothing outgrows)
    p.keep_first = batch.window > 0 ? batch.keep_first : 0;
    p.out_stride = out.row_stride != 0 ? out.row_stride : (long long)batch.nh * kD;
    p.row_scale = out.row_scale;
    p.fade_a = batch.fade_a;
    p.fade_b = batch.fade_b;
    p.out_wide = reinterpret_cast<uintptr_t>(out.out) % 32 == 0 && p.out_stride % 16 == 0 ? 1 : 0;
    p.partials = scratch.partials;
    p.counters = scratch.counters;
    CUtensorMap tmap, tmap_v;
    if (paged) {
        memcpy(&tmap, kv.tma_tile_desc, sizeof(tmap));
        memcpy(&tmap_v, static_cast<const unsigned char *>(kv.tma_tile_desc) + sizeof(tmap), sizeof(tmap_v));
    } else if (!contiguous_kv_map(&tmap, kv.k_base, kv, uint64_t(batch.const_kv_len), bf16) ||
               !contiguous_v_map(&tmap_v, kv.v_base, kv, uint64_t(batch.const_kv_len), bf16)) {
        return -1;
    }
    if (narrow(batch, kv.nkvh, grid, paged)) {
        attention_narrow_tc(stream, bf16, &tmap, &tmap_v, kv, batch, q, scale, out, scratch);
        return 0;
    }
    auto s = static_cast<cudaStream_t>(stream);
    auto run = [&](auto form) {
        constexpr int kForm = decltype(form)::value;
        bf16 ? launch<true, kForm>(s, tmap, tmap_v, p, grid, kv.overlap_launch) : launch<false, kForm>(s, tmap, tmap_v, p, grid, kv.overlap_launch);
    };
    if (p.wait_limit != kMbarWaitLimit && bf16 && !windowed) { // (a limit that tests set: by value it costs every block's waits 2 %)
        launch<true, kPlain, true>(s, tmap, tmap_v, p, grid, kv.overlap_launch);
    } else if (fading) {
        run(std::integral_constant<int, kFading>{});
    } else if (windowed) {
        run(std::integral_constant<int, kWindowed>{});
    } else {
        run(std::integral_constant<int, kPlain>{});
    }
    check_launch("paged_prefill_tc");
    return 0;
}

} // namespace llaisys::kernels
