// Recurrent mixers whose state is a matrix per head, walked CT tokens at a time on the tensor cores without giving up float32.
//
// Unrolled over a chunk, every one of these recurrences is a handful of matrix products (S0: the state at the chunk's start, for
// one head [dim keys, vdim values]; P: masked scores between the chunk's tokens; g, w: factors per token):
//     O = g_t (Q S0) + P V,        S <- decay S0 + K^T (w_s V)                     (and V <- U0 - g_t (W S0) first, for a delta rule)
// What does not depend on the state (scores, factors, W, U0) is computed by a kernel of the design's own for all chunks of a step at
// once and left in working memory (`Record`s and operand tiles); `chunk_walk_kernel` then goes from chunk to chunk.
//
// Operands.  mma.sync takes 16-bit numbers.  A float32 x is split into two halves, h = fp16(s x) and l = fp16(2^11 (s x - h)), with a
// power of two s: the numbers that one product adds up, a column's keys or tokens on the left and a token's keys or tokens on the right,
// share one s, which brings the largest of them to [2^13, 2^14); no column and no token shares it with another.  h + 2^-11 l then holds x
// to 2^-23 of itself down to 2^-28 of the largest (where h leaves fp16's normal range; below that to 2^-50 of the largest).  A product of
// two splits is h h' + 2^-11 (h l' + l h'), three instructions with float32 sums; what is left out, l l', is 2^-24 of the product.  The two
// kinds of terms have accumulators of their own, and a chunk's sums start from zero and join the state by one float32 addition, so the
// tensor cores' sums are never longer than a chunk (or than the keys of one warp).  Three products on the tensor cores (1,024
// multiply-adds a clock and multiprocessor with mma.sync, measured 960) are 2.6 times what the float32 units do (measured 122).
//
// Work.  A block owns 16 CW value columns of one (segment, head), a warp KPW keys by 16 of those columns.  It keeps the state
// transposed, as mma accumulators (rows: columns of S, columns: keys): split, they are the left operand of (Q S0)^T = S0^T Q^T without
// leaving the registers.  The warps of different keys meet in shared memory once a chunk.  Operand tiles come by bulk copies a chunk or two
// ahead (16-byte asynchronous copies by all threads took a third of a chunk's time to issue: 1,900 of 6,900 clocks for 70 KB), the
// values by 16-byte copies.
#pragma once
#include "tcgen05.cuh"
#include <cuda_fp16.h>

namespace chunk {

constexpr int CT = 32;                                    // tokens of a chunk

__device__ int walk_error = 0;                            // the library's word for a wait that ran out, where it is given no other

enum Mode { HEAD_DECAY = 0, MATRIX_MEMORY = 1, DELTA = 2, KEY_DECAY = 3 };

// ---- the split of a float32 tile into two fp16 tiles
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
constexpr float UP = 8192.f, DOWN = 1.f / 8192.f;         // what numbers of size one are scaled by
constexpr float LOW_UP = 2048.f, LOW_DOWN = 1.f / 2048.f; // what the low half is scaled by besides
// Powers of two: size <= |largest| < 2 size and up = UP / size.  (Zeros, and numbers below 2^-100: the size of 2^-100.)
struct Scale { float up, size; };
__device__ __forceinline__ Scale scale_of(unsigned largest_bits) {
    const unsigned e = min(max(largest_bits >> 23, 27u), 254u);
    return {__uint_as_float((267u - e) << 23), __uint_as_float(e << 23)};
}
__device__ __forceinline__ void split2(float a, float b, unsigned& high, unsigned& low) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((a - f.x) * LOW_UP, (b - f.y) * LOW_UP);
    high = *reinterpret_cast<const unsigned*>(&h);
    low = *reinterpret_cast<const unsigned*>(&l);
}
__device__ __forceinline__ void split1(float a, __half& high, __half& low) {
    high = __float2half_rn(a);
    low = __float2half_rn((a - __half2float(high)) * LOW_UP);
}
// the largest of what the four lanes of a row of eight (the lanes of one g) hold
__device__ __forceinline__ unsigned quad_max(unsigned x) {
    x = max(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return max(x, __shfl_xor_sync(0xffffffffu, x, 2));
}

// two floats in one register pair, for the two-at-a-time multiply-adds of sm_100
typedef unsigned long long pair;
__device__ __forceinline__ pair pair_of(float lo, float hi) {
    pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 floats_of(pair v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ pair mul2(pair a, pair b) {
    pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair fma2(pair a, pair b, pair c) {
    pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// the split of two numbers times `up`; `low_up`: up times LOW_UP
__device__ __forceinline__ void split2(pair x, pair up, pair low_up, unsigned& high, unsigned& low) {
    const float2 f = floats_of(mul2(x, up));
    const __half2 h = __floats2half2_rn(f.x, f.y);
    const float2 hf = __half22float2(h), r = floats_of(fma2(pair_of(hf.x, hf.y), pair_of(-LOW_UP, -LOW_UP), mul2(x, low_up)));
    const __half2 l = __floats2half2_rn(r.x, r.y);
    high = *reinterpret_cast<const unsigned*>(&h);
    low = *reinterpret_cast<const unsigned*>(&l);
}
// the largest magnitude of three; a NaN stays one (its bits are above infinity's)
__device__ __forceinline__ float max_abs(float a, float b, float c) {
    float r;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm(unsigned (&r)[4], const __half* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldsm_t(unsigned (&r)[4], const __half* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
// the products of two splits, without al bl, the three terms in sums of their own; and the sum of those, elements 2 i and 2 i + 1
__device__ __forceinline__ void mma3(float (&c)[3][4], const unsigned (&ah)[4], const unsigned (&al)[4], unsigned bh0, unsigned bh1, unsigned bl0,
                                     unsigned bl1) {
    mma(c[0], al, bh0, bh1);
    mma(c[1], ah, bl0, bl1);
    mma(c[2], ah, bh0, bh1);
}
__device__ __forceinline__ float2 sum3(const float (&c)[3][4], int i) {
    return make_float2(fmaf(c[0][2 * i] + c[1][2 * i], LOW_DOWN, c[2][2 * i]), fmaf(c[0][2 * i + 1] + c[1][2 * i + 1], LOW_DOWN, c[2][2 * i + 1]));
}
// ... in two sums: `main` takes the first, `cross` the other two; their sum times DOWN^2
__device__ __forceinline__ void mma3(float (&main)[4], float (&cross)[4], const unsigned (&ah)[4], const unsigned (&al)[4],
                                     unsigned bh0, unsigned bh1, unsigned bl0, unsigned bl1) {
    float p[4] = {};                                      // (the tensor cores cut their sums off; float32 additions round them)
    mma(cross, al, bh0, bh1);
    mma(p, ah, bh0, bh1);
    mma(cross, ah, bl0, bl1);
#pragma unroll
    for (int i = 0; i < 4; ++i) main[i] += p[i];
}
__device__ __forceinline__ float sum2(float main, float cross) { return fmaf(cross, LOW_DOWN, main) * (DOWN * DOWN); }

// An operand tile of CT rows of DP halves: the 16-byte group of element (row, col) lies at group (col / 8) ^ (row & 7) of its row, so
// that eight rows' groups at one column fall on different banks.
template <int DP> __device__ __forceinline__ int tile_at(int row, int col) {
    static_assert(DP % 64 == 0, "a row is whole groups of eight 16-byte groups");
    return row * DP + ((((col >> 3) ^ (row & 7)) << 3) | (col & 7));
}
// A tile of CT rows of CT halves (four groups a row).
__device__ __forceinline__ int score_at(int row, int col) { return row * CT + ((((col >> 3) ^ ((row >> 1) & 3)) << 3) | (col & 7)); }
// the left operand (16 rows by 16 columns) of such tiles
template <int DP> __device__ __forceinline__ void ldsm_left(unsigned (&r)[4], const __half* tile, int row, int col, int lane) {
    ldsm(r, tile + tile_at<DP>(row + (lane & 7) + 8 * ((lane >> 3) & 1), col + 8 * (lane >> 4)));
}
__device__ __forceinline__ void ldsm_left_scores(unsigned (&r)[4], const __half* tile, int row, int col, int lane) {
    ldsm(r, tile + score_at(row + (lane & 7) + 8 * ((lane >> 3) & 1), col + 8 * (lane >> 4)));
}

__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool on = true) {        // off: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem),
                 "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(void* smem, const void* gmem, bool on = true) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem),
                 "r"(on ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ double prefix_sum(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}
__device__ __forceinline__ double prefix_max(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = fmax(v, u);
    }
    return v;
}
// A log decay in a running sum: what lies below -1000 is as good as -1000 (any span that holds it is zero in float32), and the sum
// keeps its other terms.
__device__ __forceinline__ float bounded_log(float x) { return fmaxf(x, -1000.f); }

// ---- Which segments go in chunks: the first `segments` ones of at least `min_tokens` tokens, as far as their chunks have their places in
// working memory, which has `chunks`.  Only these segments' chunks are numbered, segment by segment: a decoded token beside a prompt's
// portion takes no memory, no block of the walk and no turn of a search.
struct Numbering { int min_tokens, chunks, segments; };
__device__ __forceinline__ int chunks_of(int tokens) { return (tokens + CT - 1) / CT; }
__device__ __forceinline__ int upto_lane(int x) {         // the sum over the lanes up to this one
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += u;
    }
    return x;
}
// The number of a segment's first chunk, or -1: it goes token by token.  All lanes of a warp ask together (in all three).
__device__ __forceinline__ int first_chunk(const Numbering& nb, const int* cu_seqlens, int seg) {
    const int tokens = cu_seqlens[seg + 1] - cu_seqlens[seg];
    if (tokens < nb.min_tokens) return -1;
    int chunks = 0, segments = 0;
    for (int s = threadIdx.x & 31; s < seg; s += 32) {
        const int n = cu_seqlens[s + 1] - cu_seqlens[s];
        if (n >= nb.min_tokens) { chunks += chunks_of(n); ++segments; }
    }
    chunks = __reduce_add_sync(0xffffffffu, chunks);
    segments = __reduce_add_sync(0xffffffffu, segments);
    return segments < nb.segments && chunks + chunks_of(tokens) <= nb.chunks ? chunks : -1;
}
// A chunk of the step: its segment, the segment's bounds, the chunk's first token and its number, or -1: its tokens are walked one by one.
struct Place { int seg, begin, end, first, at; };
// The id-th of all chunks of the step, also of those that have no number (ALL), the id-th numbered one, or the first chunk of the id-th
// segment whose chunks are (SEGMENTS); false: the step has no such chunk.
enum Search { ALL, NUMBERED, SEGMENTS };
template <int WHAT>
__device__ __forceinline__ bool find_chunk(const Numbering& nb, const int* cu_seqlens, int n_segments, int id, Place& p) {
    const int lane = threadIdx.x & 31;
    int all = 0, chunks = 0, segments = 0;                // of the segments before s0
    for (int s0 = 0; s0 < n_segments; s0 += 32) {
        const int s = s0 + lane, a = cu_seqlens[min(s, n_segments)], b = cu_seqlens[min(s + 1, n_segments)];
        const bool in = s < n_segments && b - a >= nb.min_tokens;
        const int n = chunks_of(b - a), upto_chunks = upto_lane(in ? n : 0);
        const int upto_all = WHAT == ALL ? upto_lane(n) : 0;
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        const int upto_segments = __popc(mask & (0xffffffffu >> (31 - lane)));
        const unsigned beyond = __ballot_sync(0xffffffffu, (WHAT == ALL ? all + upto_all : WHAT == NUMBERED ? chunks + upto_chunks
                                                                                                             : segments + upto_segments) > id);
        if (beyond) {
            const int src = __ffs(beyond) - 1;
            const int chunks_before = chunks + __shfl_sync(0xffffffffu, upto_chunks - (in ? n : 0), src);
            const int segments_before = segments + __shfl_sync(0xffffffffu, upto_segments - (in ? 1 : 0), src);
            const int before = WHAT == ALL ? all + __shfl_sync(0xffffffffu, upto_all - n, src) : WHAT == NUMBERED ? chunks_before : id;
            p.seg = s0 + src;
            p.begin = __shfl_sync(0xffffffffu, a, src);
            p.end = __shfl_sync(0xffffffffu, b, src);
            p.first = p.begin + (id - before) * CT;
            p.at = (mask >> src & 1) && segments_before < nb.segments && chunks_before + chunks_of(p.end - p.begin) <= nb.chunks
                       ? chunks_before + id - before : -1;
            return true;
        }
        if (WHAT == ALL) all += __shfl_sync(0xffffffffu, upto_all, 31);
        chunks += __shfl_sync(0xffffffffu, upto_chunks, 31);
        segments += __popc(mask);
    }
    return false;
}

// What a chunk needs of one head besides operand tiles (floats; double-sized parts first).  Sizes are those of the tokens' rows in the
// tiles (Scale); a row of the tile of k is divided by its size, and `w` takes it back.
//   HEAD_DECAY: g [CT], w [CT], sizes of q's rows [CT], of the scores' rows [CT], scalars [8]
//   DELTA: g, w, sizes of W's rows [CT], -, scalars (the sizes of q, k and the scores are one)
//   KEY_DECAY: -, w, sizes of q's rows, of the scores' rows, scalars, the chunk's decay per key [DP]
//   MATRIX_MEMORY: M [CT] and F [CT] as doubles, w [CT], sizes of q's rows, of the scores' rows, row sums of the scores [CT], scalars [8],
//   sum_s w_s k_s [DP]
enum Scalar { DECAY = 0, BAD = 1 };
template <int MODE, int DP> struct Record {
    static constexpr int G = 0;                           // (the memory's M, F: doubles at 0 and 2 CT)
    static constexpr int W = MODE == MATRIX_MEMORY ? 4 * CT : CT;
    static constexpr int Q_SIZE = W + CT, W_SIZE = Q_SIZE, P_SIZE = W + 2 * CT;
    static constexpr int SUMS = W + 3 * CT;               // the memory's alone
    static constexpr int SCALARS = MODE == MATRIX_MEMORY ? 8 * CT : 4 * CT;
    static constexpr int KEYS = SCALARS + 8;
    static constexpr int FLOATS = KEYS + (MODE == MATRIX_MEMORY || MODE == KEY_DECAY ? DP : 0);
    static_assert(FLOATS % 4 == 0, "records are copied in 16-byte groups");
};

// What the walk in chunks leaves to a kernel that goes token by token: short segments, and what holds numbers that are not finite (a
// masked score's zero times an infinity behind it would not be zero): a head whose operands do (`bad`, per chunk and head), or
// groups of 16 value columns whose values or state do (`columns`, [segments, heads, groups], which the walk marks as it gives them up).
struct Leftovers {
    const float* bad;                                     // null: everything is the kernel's own
    long long chunk_stride;                               // floats between two chunks' marks
    int head_stride;
    Numbering numbering;
    const int* columns; int column_groups;
};
enum Left { NOTHING = 0, MARKED_COLUMNS = 1, WHOLE = 2 };
// All threads of the block ask together, for the columns col0 .. col0 + n - 1.
__device__ __forceinline__ int left_over(const Leftovers& l, const int* cu_seqlens, int seg, int head, int heads, int col0, int n) {
    const int tokens = cu_seqlens[seg + 1] - cu_seqlens[seg];
    if (l.bad == nullptr) return WHOLE;
    const int first = first_chunk(l.numbering, cu_seqlens, seg);
    if (first < 0) return WHOLE;
    bool bad = false, marked = false;
    for (int c = threadIdx.x; c < chunks_of(tokens); c += blockDim.x)
        bad |= l.bad[(first + c) * l.chunk_stride + (long long)head * l.head_stride] != 0.f;
    const int* columns = l.columns + ((size_t)seg * heads + head) * l.column_groups;
    for (int c = col0 / 16 + threadIdx.x; c < l.column_groups && 16 * c < col0 + n; c += blockDim.x) marked |= columns[c] != 0;
    if (__syncthreads_or(bad)) return WHOLE;
    return __syncthreads_or(marked) ? MARKED_COLUMNS : NOTHING;
}
__device__ __forceinline__ bool left_column(const Leftovers& l, int what, int seg, int head, int heads, int col) {
    return what == WHOLE || l.columns[((size_t)seg * heads + head) * l.column_groups + col / 16] != 0;
}
// the marks of a segment's head, before the walk (thread `tid` of `n`)
__device__ __forceinline__ void clear_marks(int* columns, int column_groups, int seg, int head, int heads, int tid, int n) {
    for (int c = tid; c < column_groups; c += n) columns[((size_t)seg * heads + head) * column_groups + c] = 0;
}

struct Walk {
    const __half* qk;                                     // [chunks, qk_heads][q high, q low, k high, k low][CT][DP]
    const __half* w;                                      // DELTA: [chunks, heads][high, low][CT][DP]
    const __half* scores;                                 // [chunks, heads][high, low][CT][CT]
    const float* records;                                 // [chunks, heads][Record::FLOATS]
    const float* v; long long v_stride;                   // token t's values of head h: v + t v_stride + h vdim  (DELTA: U0)
    float* out; long long out_stride;                     // as v
    float* state; long long slot_stride;                  // of a slot: heads of head_stride floats
    long long head_stride;
    int key_stride, col_stride;                           // floats between two keys, two value columns of a head's state
    long long n_offset; int n_stride;                     // MATRIX_MEMORY: copies of (n, m), one for 32 columns, behind a head's state
    const float* skip;                                    // [heads]: a factor on v in the read-out, or null
    const int* cu_seqlens; const int* slots;
    int n_segments, heads, qk_heads, dim, vdim;
    float out_scale;                                      // on the read-out
    Numbering numbering;                                  // the other segments are another kernel's
    int* columns; int column_groups;                      // see Leftovers
    int stages;                                           // of the ring of chunks (2 or 3)
};

// Working memory of a step, one part after another, each on a 256-byte boundary.
struct Layout {
    long long qk, w, scores, records, u0, columns, bytes;
    int record, column_groups;
};
inline Layout layout_of(int dp, int record, int heads, int qk_heads, int vdim, int n_chunks, int n_segments, bool with_w, long long u0_floats) {
    Layout l = {};
    const auto take = [&](long long bytes) { const long long at = l.bytes; l.bytes = (at + bytes + 255) / 256 * 256; return at; };
    l.record = record;
    l.column_groups = (vdim + 15) / 16;
    l.qk = take((long long)n_chunks * qk_heads * 4 * CT * dp * 2);
    l.w = take(with_w ? (long long)n_chunks * heads * 2 * CT * dp * 2 : 0);
    l.scores = take((long long)n_chunks * heads * 2 * CT * CT * 2);
    l.records = take((long long)n_chunks * heads * record * 4);
    l.u0 = take(u0_floats * 4);
    l.columns = take((long long)n_segments * heads * l.column_groups * 4);
    return l;
}
// where the kernel before the walk leaves its results
struct Made { __half* qk; __half* w; __half* scores; float* records; float* u0; int* columns; int column_groups; Numbering numbering; };
// `n_long`: how many segments have at least min_tokens tokens, 0 if the caller does not know (each has a chunk at least)
inline Made made_at(void* scratch, const Layout& l, int min_tokens, int n_chunks, int n_segments, int n_long) {
    unsigned char* b = (unsigned char*)scratch;
    const int most = n_chunks < n_segments ? n_chunks : n_segments;
    return {(__half*)(b + l.qk), (__half*)(b + l.w), (__half*)(b + l.scores), (float*)(b + l.records), (float*)(b + l.u0),
            (int*)(b + l.columns), l.column_groups, {min_tokens, n_chunks, n_long > 0 && n_long < most ? n_long : most}};
}
inline Walk walk_of(const Made& m) {
    Walk w = {};
    w.qk = m.qk; w.w = m.w; w.scores = m.scores; w.records = m.records;
    w.columns = m.columns; w.column_groups = m.column_groups; w.numbering = m.numbering;
    w.out_scale = 1.f;
    return w;
}
inline Leftovers leftovers_of(const Made& m, const Layout& l, int heads, int scalars) {
    return {m.records + scalars + BAD, (long long)heads * l.record, l.record, m.numbering, m.columns, l.column_groups};
}

template <int KPW, int KW, int CW, int MODE> struct Shape {
    static constexpr int DP = KPW * KW, COLS = 16 * CW, THREADS = 32 * KW * CW;
    using Rec = Record<MODE, DP>;
    static constexpr int VP = COLS + 4;                   // floats of a token's row of values in shared memory
    static constexpr int TP = CT + 4;                     // floats of a column's row of sums
    static constexpr int QK_BYTES = 4 * CT * DP * 2, W_BYTES = MODE == DELTA ? 2 * CT * DP * 2 : 0, P_BYTES = 2 * CT * CT * 2;
    static constexpr int REC_BYTES = Rec::FLOATS * 4, V_BYTES = CT * VP * 4;
    static constexpr int STAGE = QK_BYTES + W_BYTES + P_BYTES + REC_BYTES + V_BYTES;
    // two sets of partial sums: in turn (a chunk's are read while the next one's are written), or a delta rule's two products
    static constexpr int SUM_FLOATS = KW * COLS * TP;
    static constexpr int SUMS = 2 * SUM_FLOATS * 4;
    // a delta rule: u, and what the read-outs start from; the memory: n and the parts of q . n of the tokens, two of each, and the tokens'
    // factors, three (a chunk's are written before its predecessor's barrier, while a slow warp may still read those of the one before)
    static constexpr int FACTORS = 3 * CT + 4;
    static constexpr int EXTRA = MODE == DELTA ? 2 * COLS * TP * 4 : MODE == MATRIX_MEMORY ? (2 * (DP + KW * CT) + 3 * FACTORS) * 4 : 0;
    static constexpr int bytes(int stages) { return stages * STAGE + SUMS + EXTRA; }
};

// What bounds it: the dependent instructions of the two warps a scheduler holds (8 x 256 x 512, 2,048 tokens: 228 us; tensor pipe 27 % of
// the time, issue slots 42 %, memory 5 %; a warp waits for the instruction before 1.5, for shared memory and shuffles 0.5, for the tensor
// pipe 0.5, at the barrier 0.3 of the 4.8 clocks between two of its instructions).  A scale per column and token instead of one a tile
// with a block-wide maximum: 201 -> 228 us; 128 x 128, 16 heads 114 -> 130; 128 x 64, 128 heads 181 -> 200; 64 x 128, 32 heads 92 -> 103.
// grid (ceil(vdim / COLS), heads, segments that go in chunks)
template <int KPW, int KW, int CW, int MODE>
__global__ void __launch_bounds__(32 * KW * CW) chunk_walk_kernel(const Walk p, const tc::WaitControl waits) {
    using SH = Shape<KPW, KW, CW, MODE>;
    using Rec = typename SH::Rec;
    constexpr int DP = SH::DP, COLS = SH::COLS, THREADS = SH::THREADS, VP = SH::VP, TP = SH::TP, NK = KPW / 8, KS = KPW / 16;
    constexpr int NT = KW >= 4 ? 1 : 4 / KW;              // groups of eight tokens whose read-outs a warp finishes
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) unsigned long long full[3];   // a stage's tiles have landed
    __shared__ int abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int kw = warp % KW, cw = warp / KW;             // the warp's keys and columns
    const int head = blockIdx.y, col0 = blockIdx.x * COLS;
    float* sums = reinterpret_cast<float*>(smem + (size_t)p.stages * SH::STAGE);
    float* extra = sums + SH::SUMS / 4;
    bool lost = false;                                    // a number that is not finite, or a wait that ran out
    int* const error_word = waits.error_word ? waits.error_word : &walk_error;
    pdl_wait();
    Place place;
    if (!find_chunk<SEGMENTS>(p.numbering, p.cu_seqlens, p.n_segments, blockIdx.z, place) || place.at < 0) return;
    const int seg = place.seg, t0 = place.begin, t1 = place.end, chunk0 = place.at;
    const int slot = p.slots[seg];
    if (seg > 0 && slot == p.slots[0]) {                  // a padding row of a captured step: its results are never read
        for (int e = tid; e < (t1 - t0) * COLS; e += THREADS)
            if (col0 + e % COLS < p.vdim) p.out[(size_t)(t0 + e / COLS) * p.out_stride + (size_t)head * p.vdim + col0 + e % COLS] = 0.f;
        return;
    }
    const int n_cols = min(COLS, p.vdim - col0), n_chunks = chunks_of(t1 - t0);
    if (tid == 0) {
        for (int i = 0; i < 3; ++i) tc::mbar_init(tc::smem_u32(&full[i]), 1);
        abort_flag = 0;
        tc::mbar_init_fence();
    }
    {
        bool bad = false;
        for (int c = tid; c < n_chunks; c += THREADS)
            bad |= p.records[((size_t)(chunk0 + c) * p.heads + head) * Rec::FLOATS + Rec::SCALARS + BAD] != 0.f;
        if (__syncthreads_or(bad)) return;
    }
    const int qk_head = head / (p.heads / p.qk_heads);
    const float* v_rows = p.v + (size_t)head * p.vdim + col0;
    const bool wide = (p.v_stride & 3) == 0 && (p.vdim & 3) == 0 && (((uintptr_t)v_rows) & 15) == 0;

    constexpr int REC_AT = SH::QK_BYTES + SH::W_BYTES + SH::P_BYTES;
    const auto fetch = [&](int c, int stage) {            // chunk c's operands into a stage
        if (c < n_chunks) {
            unsigned char* st = smem + (size_t)stage * SH::STAGE;
            if (tid == THREADS - 32) {
                const size_t at = (size_t)(chunk0 + c) * p.heads + head;
                const unsigned bar = tc::smem_u32(&full[stage]), to = tc::smem_u32(st);
                tc::mbar_expect_tx(bar, REC_AT + SH::REC_BYTES + (c == 0 ? waits.extra_tx : 0));
                tc::bulk_load(to, (const unsigned char*)p.qk + ((size_t)(chunk0 + c) * p.qk_heads + qk_head) * SH::QK_BYTES, SH::QK_BYTES, bar);
                if constexpr (MODE == DELTA) tc::bulk_load(to + SH::QK_BYTES, (const unsigned char*)p.w + at * SH::W_BYTES, SH::W_BYTES, bar);
                tc::bulk_load(to + SH::QK_BYTES + SH::W_BYTES, (const unsigned char*)p.scores + at * SH::P_BYTES, SH::P_BYTES, bar);
                tc::bulk_load(to + REC_AT, p.records + at * Rec::FLOATS, SH::REC_BYTES, bar);
            }
            float* vs = reinterpret_cast<float*>(st + REC_AT + SH::REC_BYTES);
            const int tb = t0 + c * CT, len = min(CT, t1 - tb);
            if (wide) {
                for (int e = tid; e < CT * (COLS / 4); e += THREADS) {
                    const int t = e / (COLS / 4), j = 4 * (e % (COLS / 4));
                    const bool on = t < len && j < n_cols;
                    copy16(vs + t * VP + j, on ? v_rows + (size_t)(tb + t) * p.v_stride + j : p.records, on);
                }
            } else {
                for (int e = tid; e < CT * COLS; e += THREADS) {
                    const int t = e / COLS, j = e % COLS;
                    const bool on = t < len && j < n_cols;
                    copy4(vs + t * VP + j, on ? v_rows + (size_t)(tb + t) * p.v_stride + j : p.records, on);
                }
            }
        }
        copy_commit();
    };
    // chunk c has landed, as far as this thread waits for it (another barrier makes it so for the block)
    const auto wait_for = [&](int c, int stage, unsigned parity) {
        if (p.stages > 2) copy_wait<1>(); else copy_wait<0>();
        if (c < n_chunks)
            lost |= !tc::mbar_wait(tc::smem_u32(&full[stage]), parity, &abort_flag, error_word, 2, waits.limit_cycles);
    };
    fetch(0, 0);
    if (p.stages > 2) fetch(1, 1);

    // the state's columns 16 cw + g (and + 8), keys KPW kw + 8 n + 2 t4 (and + 1)
    float* st = p.state + (size_t)slot * p.slot_stride + (size_t)head * p.head_stride;
    float S[NK][4];
    const auto state_at = [&](int n, int i, int& col, int& key) {
        col = 16 * cw + g + (i >> 1) * 8;
        key = KPW * kw + 8 * n + 2 * t4 + (i & 1);
        return col < n_cols && key < p.dim;
    };
#pragma unroll
    for (int n = 0; n < NK; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int col, key;
            S[n][i] = state_at(n, i, col, key) ? st[(size_t)key * p.key_stride + (size_t)(col0 + col) * p.col_stride] : 0.f;
        }
    const float skip = p.skip ? p.skip[head] : 0.f;
    float m_run = 0.f;                                    // MATRIX_MEMORY: the running maximum (warp 0)
    float* n_s = extra;                                   // n, then the warps' parts of q . n of the chunk's tokens
    float* nq_s = extra + 2 * DP;
    float* factors = extra + 2 * (DP + KW * CT);          // of chunk c, at c % 3: g, h, the denominator's floor [CT] each, decay, the weights' factor
    float* st_n = st + p.n_offset + (size_t)(blockIdx.x * (COLS / 32)) * p.n_stride;
    // The memory's factors per token (a lane has token `lane`): g on Q S0, h on P V.  Warp 0 makes them a chunk ahead, before a barrier
    // that every warp passes before it reads them.
    const auto make_factors = [&](const float* rec, int len, float* to) {
        const double* md = reinterpret_cast<const double*>(rec);
        const double m_local = md[lane], F = md[CT + lane];
        const double m_last = md[len - 1], F_last = md[CT + len - 1];
        const double M = fmax((double)m_run, m_local);
        to[lane] = expf((float)((double)m_run - M));
        to[CT + lane] = expf((float)(m_local - M));
        to[2 * CT + lane] = expf(-(float)(F + M));
        // the maximum goes on as a float, and the state is scaled to that rounded value
        const float m_next = (float)(F_last + fmax((double)m_run, m_last));
        const double M_state = (double)m_next - F_last;
        if (lane == 0) {
            to[3 * CT] = expf((float)((double)m_run - M_state));
            to[3 * CT + 1] = expf((float)(m_last - M_state));
        }
        m_run = m_next;
    };
    if constexpr (MODE == MATRIX_MEMORY) {
        static_assert(COLS % 32 == 0, "a copy of n serves 32 columns");
        if (warp == 0) m_run = st_n[p.dim];
        for (int d = tid; d < DP; d += THREADS) n_s[d] = d < p.dim ? st_n[d] : 0.f;
    }
    wait_for(0, 0, 0);
    __syncthreads();
    if constexpr (MODE == MATRIX_MEMORY) {
        if (warp == 0) make_factors(reinterpret_cast<const float*>(smem + REC_AT), min(CT, t1 - t0), factors);
        __syncthreads();
    }
    // where a lane reads the operand tiles (halves from a tile's start), whatever the chunk
    int at_q[KS];
#pragma unroll
    for (int k = 0; k < KS; ++k) at_q[k] = tile_at<DP>(8 * (lane >> 4) + (lane & 7), KPW * kw + 16 * k + 8 * ((lane >> 3) & 1));

    int stage = 0;                                        // of chunk c
    unsigned parity = 0, slot3 = 0;                       // of the stage's barrier for chunk c; c % 3
    int c = 0;
#pragma unroll 1
    for (; c < n_chunks; ++c) {
        // (into the stage of the chunk before, which every warp has left)
        fetch(c + p.stages - 1, stage == 0 ? p.stages - 1 : stage - 1);
        unsigned char* stg = smem + (size_t)stage * SH::STAGE;
        if (++stage == p.stages) { stage = 0; parity ^= 1; }          // (of the next chunk from here on)
        const __half* q_s = reinterpret_cast<const __half*>(stg);
        const __half* k_s = q_s + 2 * CT * DP;
        const __half* w_s = k_s + 2 * CT * DP;
        const __half* p_s = reinterpret_cast<const __half*>(stg + SH::QK_BYTES + SH::W_BYTES);
        const float* rec = reinterpret_cast<const float*>(stg + REC_AT);
        const float* v_s = reinterpret_cast<const float*>(stg + REC_AT + SH::REC_BYTES);
        const int tb = t0 + c * CT, len = min(CT, t1 - tb);
        float* sum = sums + (MODE == DELTA ? 0 : (c & 1) * SH::SUM_FLOATS);
        const float* fac = factors + slot3 * SH::FACTORS;
        const unsigned slot_next = slot3 == 2 ? 0 : slot3 + 1;

        // ---- (Q S0)^T, and (W S0)^T, over the warp's keys: still to be multiplied by the sizes of q's and W's rows
        {
            float largest[2] = {0.f, 0.f}, down[2];       // of the columns g and g + 8
            pair up[2], low_up[2];
#pragma unroll
            for (int n = 0; n < NK; ++n)
#pragma unroll
                for (int i = 0; i < 2; ++i) largest[i] = max_abs(largest[i], S[n][2 * i], S[n][2 * i + 1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned bits = quad_max(__float_as_uint(largest[i]));
                lost |= bits >= 0x7f800000u;
                const Scale s = scale_of(bits);
                up[i] = pair_of(s.up, s.up);
                low_up[i] = pair_of(s.up * LOW_UP, s.up * LOW_UP);
                down[i] = s.size * (DOWN * DOWN);
            }
            unsigned ah[KS][4], al[KS][4];
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    split2(pair_of(S[2 * k + (i >> 1)][2 * (i & 1)], S[2 * k + (i >> 1)][2 * (i & 1) + 1]), up[i & 1], low_up[i & 1], ah[k][i], al[k][i]);
            const auto product = [&](const __half* tile, float* to) {
                to += (kw * COLS + 16 * cw + g) * TP + 2 * t4;
                float acc[4][3][4] = {};                  // groups of eight tokens; the terms apart, so that no sum waits for another
#pragma unroll
                for (int k = 0; k < KS; ++k)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        unsigned bh[4], bl[4];
                        ldsm(bh, tile + at_q[k] + half * 16 * DP);
                        ldsm(bl, tile + CT * DP + at_q[k] + half * 16 * DP);
                        mma3(acc[2 * half], ah[k], al[k], bh[0], bh[1], bl[0], bl[1]);
                        mma3(acc[2 * half + 1], ah[k], al[k], bh[2], bh[3], bl[2], bl[3]);
                    }
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float2 x = sum3(acc[n], i);
                        *(float2*)(to + 8 * i * TP + 8 * n) = make_float2(x.x * down[i], x.y * down[i]);
                    }
            };
            product(q_s, sum);
            if constexpr (MODE == DELTA) product(w_s, sum + SH::SUM_FLOATS);
        }
        // ---- the chunk's values as left operands (columns g, g + 8; tokens 16 k + 2 t4, + 1, + 8, + 9)
        float2 va[2][4];                                  // [sixteen tokens][register]
        if constexpr (MODE == DELTA) {                    // V <- U0 - g (W S0); what the read-outs start from beside it
            __syncthreads();
            float* u_s = extra;
            float* z_s = extra + COLS * TP;
            for (int e = tid; e < COLS * (CT / 4); e += THREADS) {
                const int j = e % COLS, t = 4 * (e / COLS);
                float4 y = make_float4(0.f, 0.f, 0.f, 0.f), z = y;
#pragma unroll
                for (int k = 0; k < KW; ++k) {
                    const float4 a = *(const float4*)(sum + (k * COLS + j) * TP + t), b = *(const float4*)(sum + SH::SUM_FLOATS + (k * COLS + j) * TP + t);
                    z.x += a.x; z.y += a.y; z.z += a.z; z.w += a.w;
                    y.x += b.x; y.y += b.y; y.z += b.z; y.w += b.w;
                }
                const float4 gg = *(const float4*)(rec + Rec::G + t), ws = *(const float4*)(rec + Rec::W_SIZE + t);
                *(float4*)(u_s + j * TP + t) =
                    make_float4(fmaf(-gg.x, y.x * ws.x, v_s[t * VP + j]), fmaf(-gg.y, y.y * ws.y, v_s[(t + 1) * VP + j]),
                                fmaf(-gg.z, y.z * ws.z, v_s[(t + 2) * VP + j]), fmaf(-gg.w, y.w * ws.w, v_s[(t + 3) * VP + j]));
                *(float4*)(z_s + j * TP + t) = make_float4(gg.x * z.x, gg.y * z.y, gg.z * z.z, gg.w * z.w);
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) va[k][i] = *(const float2*)(u_s + (16 * cw + g + 8 * (i & 1)) * TP + 16 * k + 2 * t4 + 8 * (i >> 1));
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float* v = v_s + (16 * k + 2 * t4 + 8 * (i >> 1)) * VP + 16 * cw + g + 8 * (i & 1);
                    va[k][i] = make_float2(v[0], v[VP]);
                }
        }
        unsigned vh[2][4], vl[2][4];                      // V split, and as it joins the state
        float v_down[2];                                  // the columns' sizes times DOWN^2
        const auto split_values = [&] {
            pair up[2], low_up[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float m = max_abs(max_abs(max_abs(va[0][i].x, va[0][i].y, va[0][i + 2].x), va[0][i + 2].y, va[1][i].x),
                                        max_abs(va[1][i].y, va[1][i + 2].x, va[1][i + 2].y), 0.f);
                const unsigned bits = quad_max(__float_as_uint(m));
                lost |= bits >= 0x7f800000u;
                const Scale s = scale_of(bits);
                up[i] = pair_of(s.up, s.up);
                low_up[i] = pair_of(s.up * LOW_UP, s.up * LOW_UP);
                v_down[i] = s.size * (DOWN * DOWN);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) split2(pair_of(va[k][i].x, va[k][i].y), up[i & 1], low_up[i & 1], vh[k][i], vl[k][i]);
        };
        split_values();
        // ---- P V of the tokens that the warp finishes (still to be multiplied by the sizes of P's rows)
        float o[NT][4];
        if (KW <= 4 || kw < 4) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float acc[3][4] = {};
                const int row = 8 * (NT * kw + n) + (lane & 7);
                unsigned bh[4], bl[4];                    // the four groups of eight tokens s
                ldsm(bh, p_s + score_at(row, 8 * (lane >> 3)));
                ldsm(bl, p_s + CT * CT + score_at(row, 8 * (lane >> 3)));
                mma3(acc, vh[0], vl[0], bh[0], bh[1], bl[0], bl[1]);
                mma3(acc, vh[1], vl[1], bh[2], bh[3], bl[2], bl[3]);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 x = sum3(acc, r);
                    o[n][2 * r] = x.x * v_down[r]; o[n][2 * r + 1] = x.y * v_down[r];
                }
            }
        }
        // ---- the state after the chunk
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 w = *(const float2*)(rec + Rec::W + 16 * k + 2 * t4 + 8 * (i >> 1));
                va[k][i].x *= w.x; va[k][i].y *= w.y;
            }
        split_values();
        {
            float decay;
            if constexpr (MODE == MATRIX_MEMORY) { decay = fac[3 * CT]; v_down[0] *= fac[3 * CT + 1]; v_down[1] *= fac[3 * CT + 1]; }
            else decay = rec[Rec::SCALARS + DECAY];
            const pair down2[2] = {pair_of(v_down[0], v_down[0]), pair_of(v_down[1], v_down[1])};
            pair decay2 = pair_of(decay, decay);
            constexpr int NB = NK < 4 ? NK : 4;           // groups of eight keys at a time
#pragma unroll
            for (int n = 0; n < NK; n += NB) {
                float acc[NB][3][4] = {};
#pragma unroll
                for (int k = 0; k < 2; ++k)
#pragma unroll
                    for (int j = 0; j < NB / 2; ++j) {
                        const int at = tile_at<DP>(16 * k + 8 * ((lane >> 3) & 1) + (lane & 7), KPW * kw + 8 * (n + 2 * j) + 8 * (lane >> 4));
                        unsigned bh[4], bl[4];
                        ldsm_t(bh, k_s + at);
                        ldsm_t(bl, k_s + CT * DP + at);
                        mma3(acc[2 * j], vh[k], vl[k], bh[0], bh[1], bl[0], bl[1]);
                        mma3(acc[2 * j + 1], vh[k], vl[k], bh[2], bh[3], bl[2], bl[3]);
                    }
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    if constexpr (MODE == KEY_DECAY) {
                        const float2 d = *(const float2*)(rec + Rec::KEYS + KPW * kw + 8 * (n + j) + 2 * t4);
                        decay2 = pair_of(d.x, d.y);
                    }
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const float2 y = sum3(acc[j], r);
                        const float2 x = floats_of(fma2(decay2, pair_of(S[n + j][2 * r], S[n + j][2 * r + 1]), mul2(pair_of(y.x, y.y), down2[r])));
                        S[n + j][2 * r] = x.x; S[n + j][2 * r + 1] = x.y;
                    }
                }
            }
        }
        slot3 = slot_next;
        if constexpr (MODE == MATRIX_MEMORY) {
            // q . n of sixteen tokens over the warp's keys (n is row 0 of a left operand), then n after the chunk
            const float* n_old = n_s + (c & 1) * DP;
            float* n_new = n_s + ((c + 1) & 1) * DP;
            if (cw < 2) {
                float acc[2][3][4] = {};
                float2 x[KS][2];
                float m = 0.f;
#pragma unroll
                for (int k = 0; k < KS; ++k)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        x[k][i] = g == 0 ? *(const float2*)(n_old + KPW * kw + 16 * k + 8 * i + 2 * t4) : make_float2(0.f, 0.f);
                        m = max_abs(m, x[k][i].x, x[k][i].y);
                    }
                const unsigned bits = quad_max(__float_as_uint(m));
                lost |= bits >= 0x7f800000u;
                const Scale sn = scale_of(bits);
                const pair up = pair_of(sn.up, sn.up), low_up = pair_of(sn.up * LOW_UP, sn.up * LOW_UP);
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    unsigned ah[4] = {}, al[4] = {}, bh[4], bl[4];
                    if (g == 0) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) split2(pair_of(x[k][i].x, x[k][i].y), up, low_up, ah[2 * i], al[2 * i]);
                    }
                    ldsm(bh, q_s + at_q[k] + cw * 16 * DP);
                    ldsm(bl, q_s + CT * DP + at_q[k] + cw * 16 * DP);
                    mma3(acc[0], ah, al, bh[0], bh[1], bl[0], bl[1]);
                    mma3(acc[1], ah, al, bh[2], bh[3], bl[2], bl[3]);
                }
                if (g == 0) {
                    float* to = nq_s + ((c & 1) * KW + kw) * CT + 16 * cw + 2 * t4;
                    const float down = sn.size * (DOWN * DOWN);          // (still to be multiplied by the sizes of q's rows)
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        const float2 y = sum3(acc[n], 0);
                        *(float2*)(to + 8 * n) = make_float2(y.x * down, y.y * down);
                    }
                }
            }
            for (int d = tid; d < DP; d += THREADS) n_new[d] = fmaf(fac[3 * CT], n_old[d], fac[3 * CT + 1] * rec[Rec::KEYS + d]);
        }
        wait_for(c + 1, stage, parity);
        if constexpr (MODE == MATRIX_MEMORY) {            // the next chunk's factors, in front of the barrier below
            if (warp == 0 && c + 1 < n_chunks)
                make_factors(reinterpret_cast<const float*>(smem + (size_t)stage * SH::STAGE + REC_AT), min(CT, t1 - tb - CT),
                             factors + slot_next * SH::FACTORS);
        }
        // what the read-outs take from this chunk's stage
        float2 gt[NT], row_sum[NT], skipped[NT][2], q_size[NT], p_size[NT];
        if constexpr (MODE != DELTA) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int t = 8 * (NT * kw + n) + 2 * t4;
                q_size[n] = *(const float2*)(rec + Rec::Q_SIZE + (t & 31));
                p_size[n] = *(const float2*)(rec + Rec::P_SIZE + (t & 31));
                if constexpr (MODE == HEAD_DECAY) {
                    gt[n] = *(const float2*)(rec + Rec::G + (t & 31));
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        skipped[n][r] = make_float2(skip * v_s[t * VP + 16 * cw + g + 8 * r], skip * v_s[(t + 1) * VP + 16 * cw + g + 8 * r]);
                }
                if constexpr (MODE == MATRIX_MEMORY) {
                    gt[n] = *(const float2*)(fac + (t & 31));
                    row_sum[n] = *(const float2*)(rec + Rec::SUMS + (t & 31));
                }
            }
            lost = __syncthreads_or(lost);                // the sums over the keys are complete, and this chunk's stage is free
            if (lost) break;
        }
        if (KW <= 4 || kw < 4) {
            float* out = p.out + (size_t)tb * p.out_stride + (size_t)head * p.vdim + col0;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int t = 8 * (NT * kw + n) + 2 * t4;
                float2 fz = make_float2(p.out_scale, p.out_scale), fo = fz;
                if constexpr (MODE != DELTA) {
                    fz.x *= q_size[n].x; fz.y *= q_size[n].y; fo.x *= p_size[n].x; fo.y *= p_size[n].y;
                }
                if constexpr (MODE == HEAD_DECAY) { fz.x *= gt[n].x; fz.y *= gt[n].y; }
                if constexpr (MODE == MATRIX_MEMORY) {
                    const float2 ht = *(const float2*)(fac + CT + t), floor = *(const float2*)(fac + 2 * CT + t);
                    float2 nq = make_float2(0.f, 0.f);
#pragma unroll
                    for (int k = 0; k < KW; ++k) {
                        const float2 a = *(const float2*)(nq_s + ((c & 1) * KW + k) * CT + t);
                        nq.x += a.x; nq.y += a.y;
                    }
                    nq.x *= q_size[n].x; nq.y *= q_size[n].y;
                    const float rx = 1.f / (fmaxf(fabsf(p.out_scale * (gt[n].x * nq.x + ht.x * row_sum[n].x)), floor.x) + 1e-6f);
                    const float ry = 1.f / (fmaxf(fabsf(p.out_scale * (gt[n].y * nq.y + ht.y * row_sum[n].y)), floor.y) + 1e-6f);
                    fz.x *= gt[n].x * rx; fz.y *= gt[n].y * ry; fo.x *= ht.x * rx; fo.y *= ht.y * ry;
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int col = 16 * cw + g + 8 * r;
                    float2 x;
                    if constexpr (MODE == DELTA) {
                        const float2 z = *(const float2*)(extra + (COLS + col) * TP + t);
                        x = make_float2(fmaf(fo.x, o[n][2 * r], p.out_scale * z.x), fmaf(fo.y, o[n][2 * r + 1], p.out_scale * z.y));
                    } else {
                        float2 z = make_float2(0.f, 0.f);
#pragma unroll
                        for (int k = 0; k < KW; ++k) {
                            const float2 a = *(const float2*)(sum + (k * COLS + col) * TP + t);
                            z.x += a.x; z.y += a.y;
                        }
                        x = make_float2(fmaf(fz.x, z.x, fo.x * o[n][2 * r]), fmaf(fz.y, z.y, fo.y * o[n][2 * r + 1]));
                        if constexpr (MODE == HEAD_DECAY) { x.x += skipped[n][r].x; x.y += skipped[n][r].y; }
                    }
                    if (col < n_cols) {
                        if (t < len) out[(size_t)t * p.out_stride + col] = x.x;
                        if (t + 1 < len) out[(size_t)(t + 1) * p.out_stride + col] = x.y;
                    }
                }
            }
        }
        if constexpr (MODE == DELTA) {                    // (the stage, the sums and u are free)
            lost = __syncthreads_or(lost);
            if (lost) break;
        }
    }
    copy_wait<0>();
    if (lost) {                                           // the slot is as it was, and the columns go token by token
        if (tid == 0)                                     // (copies in flight land before the block leaves: chunk c's too, whose wait may
            for (int x = c; x < min(c + p.stages, n_chunks); ++x)          // be the one that ran out)
                tc::mbar_drain(tc::smem_u32(&full[x % p.stages]), (x / p.stages) & 1, waits.limit_cycles);
        __syncthreads();
        if (tid < CW && col0 / 16 + tid < p.column_groups) p.columns[((size_t)seg * p.heads + head) * p.column_groups + col0 / 16 + tid] = 1;
        return;
    }
#pragma unroll
    for (int n = 0; n < NK; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int col, key;
            if (state_at(n, i, col, key)) st[(size_t)key * p.key_stride + (size_t)(col0 + col) * p.col_stride] = S[n][i];
        }
    if constexpr (MODE == MATRIX_MEMORY) {
        __syncthreads();
        for (int b = 0; b < COLS / 32 && col0 + 32 * b < p.vdim; ++b) {
            for (int d = tid; d < p.dim; d += THREADS) st_n[(size_t)b * p.n_stride + d] = n_s[(n_chunks & 1) * DP + d];
            if (tid == 0) st_n[(size_t)b * p.n_stride + p.dim] = m_run;
        }
    }
}

template <int KPW, int KW, int CW, int MODE>
int launch_walk(Walk p, const tc::WaitControl& waits, cudaStream_t st) {
    using SH = Shape<KPW, KW, CW, MODE>;
    dim3 grid((p.vdim + SH::COLS - 1) / SH::COLS, p.heads, p.numbering.segments);
    // three stages where a multiprocessor holds one block anyway, two where two blocks then fit
    constexpr bool three = SH::bytes(3) <= 227 * 1024;
    p.stages = three && (long long)grid.x * grid.y * grid.z <= 148 ? 3 : 2;
    auto kernel = chunk_walk_kernel<KPW, KW, CW, MODE>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::bytes(three ? 3 : 2)) != cudaSuccess)
        return SPITE_LAUNCH_FAILED;
    // (in the ordinary way: started early, the blocks would sit on the multiprocessors of the kernel before, several to one)
    kernel<<<grid, SH::THREADS, SH::bytes(p.stages), st>>>(p, waits);
    return spite_launch_status();
}

}  // namespace chunk
