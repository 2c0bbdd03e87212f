// Recurrent mixers whose state is a matrix per head, walked CT tokens at a time on the tensor cores without giving up float32.
//
// Unrolled over a chunk, every one of these recurrences is a handful of matrix products (S0: the state at the chunk's start, for
// one head [dim keys, vdim values]; P: masked scores between the chunk's tokens; g, w: factors per token):
//     O = g_t (Q S0) + P V,        S <- decay S0 + K^T (w_s V)                     (and V <- U0 - g_t (W S0) first, for a delta rule)
// What does not depend on the state (scores, factors, W, U0) is computed by a kernel of the design's own for all chunks of a step at
// once and left in working memory (`Record`s and operand tiles); `chunk_walk_kernel` then goes from chunk to chunk.
//
// Operands.  mma.sync takes 16-bit numbers.  A float32 x is split into two halves, h = fp16(s x) and l = fp16(s x - h), with a power of
// two s that brings the tile's largest element to [2^13, 2^14): h + l then holds x to 2^-23 of itself (and no worse than 2^-38 of the
// tile's largest element, where l leaves fp16's normal range), and a product of two splits is h h' + (h l' + l h'), three
// instructions with float32 sums; what is left out, l l', is 2^-24 of the product.  The two kinds of terms have accumulators of
// their own, and a chunk's sums start from zero and join the state by one float32 addition, so the tensor cores' sums are never
// longer than a chunk (or than the keys of one warp).  Three products on the tensor cores (1,024 multiply-adds a clock and
// multiprocessor with mma.sync, measured 960) are 2.6 times what the float32 units do (measured 122).
//
// Work.  A block owns 16 CW value columns of one (segment, head), a warp KPW keys by 16 of those columns.  It keeps the state
// transposed, as mma accumulators (rows: columns of S, columns: keys): split, they are the left operand of (Q S0)^T = S0^T Q^T without
// leaving the registers.  The warps of different keys meet in shared memory once a chunk.  Operand tiles and values come by asynchronous
// copies a chunk or two ahead.
#pragma once
#include "common.cuh"
#include <cuda_fp16.h>

namespace chunk {

constexpr int CT = 32;                                    // tokens of a chunk

enum Mode { HEAD_DECAY = 0, MATRIX_MEMORY = 1, DELTA = 2, KEY_DECAY = 3 };

// ---- the split of a float32 tile into two fp16 tiles
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
struct Scale { float up, down; };                         // powers of two, up * down = 1
__device__ __forceinline__ Scale scale_of(unsigned largest_bits) {
    const unsigned e = min(max(largest_bits >> 23, 14u), 254u);       // (a tile of zeros, or of numbers below 2^-113: the largest factor)
    return {__uint_as_float((267u - e) << 23), __uint_as_float((e - 13u) << 23)};
}
__device__ __forceinline__ void split2(float a, float b, unsigned& high, unsigned& low) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    high = *reinterpret_cast<const unsigned*>(&h);
    low = *reinterpret_cast<const unsigned*>(&l);
}
__device__ __forceinline__ void split1(float a, __half& high, __half& low) {
    high = __float2half_rn(a);
    low = __float2half_rn(a - __half2float(high));
}

__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
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
// c += (ah + al)(bh + bl) without al bl: `main` takes the first, `cross` the other two
__device__ __forceinline__ void mma3(float (&main)[4], float (&cross)[4], const unsigned (&ah)[4], const unsigned (&al)[4],
                                     unsigned bh0, unsigned bh1, unsigned bl0, unsigned bl1) {
    mma(cross, al, bh0, bh1);
    mma(main, ah, bh0, bh1);
    mma(cross, ah, bl0, bl1);
}

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

// ---- chunks are numbered segment by segment
__device__ __forceinline__ int chunks_before(const int* cu_seqlens, int seg) {
    int n = 0;
    for (int s = 0; s < seg; ++s) n += (cu_seqlens[s + 1] - cu_seqlens[s] + CT - 1) / CT;
    return n;
}
// the segment of a chunk and the chunk's first token; false: the step has no such chunk
__device__ __forceinline__ bool find_chunk(const int* cu_seqlens, int n_segments, int id, int& seg, int& first) {
    for (seg = 0; seg < n_segments; ++seg) {
        const int n = (cu_seqlens[seg + 1] - cu_seqlens[seg] + CT - 1) / CT;
        if (id < n) { first = cu_seqlens[seg] + id * CT; return true; }
        id -= n;
    }
    return false;
}

// What a chunk needs of one head besides operand tiles (floats; double-sized parts first).
//   HEAD_DECAY, DELTA, KEY_DECAY: g [CT], w [CT], scalars [8]   (KEY_DECAY: and the chunk's decay per key [DP])
//   MATRIX_MEMORY: M [CT] and F [CT] as doubles, w [CT], row sums of the scores [CT], scalars [8], sum_s w_s k_s [DP]
enum Scalar { Q_DOWN = 0, K_DOWN = 1, P_DOWN = 2, DECAY = 3, W_DOWN = 4, BAD = 5 };
template <int MODE, int DP> struct Record {
    static constexpr int G = 0;                           // (the memory's M, F: doubles at 0 and 2 CT)
    static constexpr int W = MODE == MATRIX_MEMORY ? 4 * CT : CT;
    static constexpr int SUMS = 5 * CT;                   // the memory's alone
    static constexpr int SCALARS = MODE == MATRIX_MEMORY ? 6 * CT : 2 * CT;
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
    int head_stride, min_tokens;
    const int* columns; int column_groups;
};
enum Left { NOTHING = 0, MARKED_COLUMNS = 1, WHOLE = 2 };
// All threads of the block ask together, for the columns col0 .. col0 + n - 1.
__device__ __forceinline__ int left_over(const Leftovers& l, const int* cu_seqlens, int seg, int head, int heads, int col0, int n) {
    const int tokens = cu_seqlens[seg + 1] - cu_seqlens[seg];
    if (l.bad == nullptr || tokens < l.min_tokens) return WHOLE;
    const int first = chunks_before(cu_seqlens, seg);
    bool bad = false, marked = false;
    for (int c = threadIdx.x; c < (tokens + CT - 1) / CT; c += blockDim.x)
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
    int min_tokens;                                       // shorter segments are another kernel's
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
struct Made { __half* qk; __half* w; __half* scores; float* records; float* u0; int* columns; int column_groups, min_tokens; };
inline Made made_at(void* scratch, const Layout& l, int min_tokens) {
    unsigned char* b = (unsigned char*)scratch;
    return {(__half*)(b + l.qk), (__half*)(b + l.w), (__half*)(b + l.scores), (float*)(b + l.records), (float*)(b + l.u0),
            (int*)(b + l.columns), l.column_groups, min_tokens};
}
inline Walk walk_of(const Made& m) {
    Walk w = {};
    w.qk = m.qk; w.w = m.w; w.scores = m.scores; w.records = m.records;
    w.columns = m.columns; w.column_groups = m.column_groups; w.min_tokens = m.min_tokens;
    w.out_scale = 1.f;
    return w;
}
inline Leftovers leftovers_of(const Made& m, const Layout& l, int heads, int scalars) {
    return {m.records + scalars + BAD, (long long)heads * l.record, l.record, m.min_tokens, m.columns, l.column_groups};
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
    static constexpr int EXTRA = MODE == DELTA ? 2 * COLS * TP * 4 : MODE == MATRIX_MEMORY ? (2 * DP + 2 * CT) * 4 : 0;
    static constexpr int bytes(int stages) { return stages * STAGE + SUMS + EXTRA; }
};

// grid (ceil(vdim / COLS), heads, segments)
template <int KPW, int KW, int CW, int MODE>
__global__ void __launch_bounds__(32 * KW * CW) chunk_walk_kernel(const Walk p) {
    using SH = Shape<KPW, KW, CW, MODE>;
    using Rec = typename SH::Rec;
    constexpr int DP = SH::DP, COLS = SH::COLS, THREADS = SH::THREADS, VP = SH::VP, TP = SH::TP, NK = KPW / 8, KS = KPW / 16;
    constexpr int NT = KW >= 4 ? 1 : 4 / KW;              // groups of eight tokens whose read-outs a warp finishes
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int kw = warp % KW, cw = warp / KW;             // the warp's keys and columns
    const int seg = blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * COLS;
    float* sums = reinterpret_cast<float*>(smem + (size_t)p.stages * SH::STAGE);
    float* extra = sums + SH::SUMS / 4;
    bool lost = false;                                    // a number that is not finite
    pdl_wait();
    const int t0 = p.cu_seqlens[seg], t1 = p.cu_seqlens[seg + 1];
    if (t1 - t0 < p.min_tokens) return;
    const int slot = p.slots[seg];
    if (seg > 0 && slot == p.slots[0]) {                  // a padding row of a captured step: its results are never read
        for (int e = tid; e < (t1 - t0) * COLS; e += THREADS)
            if (col0 + e % COLS < p.vdim) p.out[(size_t)(t0 + e / COLS) * p.out_stride + (size_t)head * p.vdim + col0 + e % COLS] = 0.f;
        return;
    }
    const int n_cols = min(COLS, p.vdim - col0), n_chunks = (t1 - t0 + CT - 1) / CT, chunk0 = chunks_before(p.cu_seqlens, seg);
    {
        bool bad = false;
        for (int c = tid; c < n_chunks; c += THREADS)
            bad |= p.records[((size_t)(chunk0 + c) * p.heads + head) * Rec::FLOATS + Rec::SCALARS + BAD] != 0.f;
        if (__syncthreads_or(bad)) return;
    }
    const int qk_head = head / (p.heads / p.qk_heads);
    const float* v_rows = p.v + (size_t)head * p.vdim + col0;
    const bool wide = (p.v_stride & 3) == 0 && (p.vdim & 3) == 0 && (((uintptr_t)v_rows) & 15) == 0;

    const auto fetch = [&](int c) {                       // the chunk's operands into its stage
        if (c < n_chunks) {
            unsigned char* st = smem + (size_t)(c % p.stages) * SH::STAGE;
            const size_t at = (size_t)(chunk0 + c) * p.heads + head;
            const unsigned char* qk = (const unsigned char*)p.qk + ((size_t)(chunk0 + c) * p.qk_heads + qk_head) * SH::QK_BYTES;
#pragma unroll 4
            for (int e = tid * 16; e < SH::QK_BYTES; e += THREADS * 16) copy16(st + e, qk + e);
            if constexpr (MODE == DELTA) {
                const unsigned char* w = (const unsigned char*)p.w + at * SH::W_BYTES;
#pragma unroll 4
                for (int e = tid * 16; e < SH::W_BYTES; e += THREADS * 16) copy16(st + SH::QK_BYTES + e, w + e);
            }
            unsigned char* rest = st + SH::QK_BYTES + SH::W_BYTES;
            const unsigned char* sc = (const unsigned char*)p.scores + at * SH::P_BYTES;
            const unsigned char* rec = (const unsigned char*)(p.records + at * Rec::FLOATS);
            for (int e = tid * 16; e < SH::P_BYTES; e += THREADS * 16) copy16(rest + e, sc + e);
            for (int e = tid * 16; e < SH::REC_BYTES; e += THREADS * 16) copy16(rest + SH::P_BYTES + e, rec + e);
            float* vs = reinterpret_cast<float*>(rest + SH::P_BYTES + SH::REC_BYTES);
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
    fetch(0);
    if (p.stages > 2) fetch(1);

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
    float m_run = 0.f;
    float* n_s = extra;                                   // MATRIX_MEMORY: n, two copies in turn, then q . n of the chunk's tokens
    float* st_n = st + p.n_offset + (size_t)(blockIdx.x * (COLS / 32)) * p.n_stride;
    if constexpr (MODE == MATRIX_MEMORY) {
        static_assert(COLS % 32 == 0, "a copy of n serves 32 columns");
        m_run = st_n[p.dim];
        for (int d = tid; d < DP; d += THREADS) n_s[d] = d < p.dim ? st_n[d] : 0.f;
    }
    if (p.stages > 2) copy_wait<1>(); else copy_wait<0>();
    __syncthreads();

#pragma unroll 1
    for (int c = 0; c < n_chunks; ++c) {
        fetch(c + p.stages - 1);                          // (into the stage of the chunk before, which every warp has left)
        unsigned char* stg = smem + (size_t)(c % p.stages) * SH::STAGE;
        const __half* q_s = reinterpret_cast<const __half*>(stg);
        const __half* k_s = q_s + 2 * CT * DP;
        const __half* w_s = k_s + 2 * CT * DP;
        const __half* p_s = reinterpret_cast<const __half*>(stg + SH::QK_BYTES + SH::W_BYTES);
        const float* rec = reinterpret_cast<const float*>(stg + SH::QK_BYTES + SH::W_BYTES + SH::P_BYTES);
        const float* v_s = reinterpret_cast<const float*>(stg + SH::QK_BYTES + SH::W_BYTES + SH::P_BYTES + SH::REC_BYTES);
        const int tb = t0 + c * CT, len = min(CT, t1 - tb);
        float* sum = sums + (MODE == DELTA ? 0 : (c & 1) * SH::SUM_FLOATS);

        // factors per token (a lane has token `lane`): g on Q S0, h on P V, w on V in the state's renewal
        float gt, ht = 1.f, wt, decay, den = 1.f, w_more = 1.f;
        if constexpr (MODE == MATRIX_MEMORY) {
            const double* md = reinterpret_cast<const double*>(rec);
            const double m_local = md[lane], F = md[CT + lane];
            const double m_last = md[len - 1], F_last = md[CT + len - 1];
            const double M = fmax((double)m_run, m_local);
            gt = expf((float)((double)m_run - M));
            ht = expf((float)(m_local - M));
            // the maximum goes on as a float, and the state is scaled to that rounded value
            const float m_next = (float)(F_last + fmax((double)m_run, m_last));
            const double M_state = (double)m_next - F_last;
            w_more = expf((float)(m_last - M_state));
            wt = rec[Rec::W + lane] * w_more;
            decay = expf((float)((double)m_run - M_state));
            den = expf(-(float)(F + M));
            m_run = m_next;
        } else {
            gt = rec[Rec::G + lane];
            wt = rec[Rec::W + lane];
            decay = rec[Rec::SCALARS + DECAY];
        }
        const float q_down = rec[Rec::SCALARS + Q_DOWN], k_down = rec[Rec::SCALARS + K_DOWN], p_down = rec[Rec::SCALARS + P_DOWN];

        // ---- (Q S0)^T, and (W S0)^T, over the warp's keys
        {
            unsigned largest = 0;
#pragma unroll
            for (int n = 0; n < NK; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) largest = max(largest, abs_bits(S[n][i]));
            largest = __reduce_max_sync(0xffffffffu, largest);
            lost |= largest >= 0x7f800000u;
            const Scale s = scale_of(largest);
            unsigned ah[KS][4], al[KS][4];
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    split2(S[2 * k + (i >> 1)][2 * (i & 1)] * s.up, S[2 * k + (i >> 1)][2 * (i & 1) + 1] * s.up, ah[k][i], al[k][i]);
            const auto product = [&](const __half* tile, float down, float* to) {
                to += (kw * COLS + 16 * cw + g) * TP + 2 * t4;
#pragma unroll
                for (int half = 0; half < 2; ++half) {    // sixteen tokens at a time
                    float main[2][4] = {}, cross[2][4] = {};
#pragma unroll
                    for (int k = 0; k < KS; ++k) {
                        const int row = 16 * half + 8 * (lane >> 4) + (lane & 7), col = KPW * kw + 16 * k + 8 * ((lane >> 3) & 1);
                        unsigned bh[4], bl[4];
                        ldsm(bh, tile + tile_at<DP>(row, col));
                        ldsm(bl, tile + CT * DP + tile_at<DP>(row, col));
                        mma3(main[0], cross[0], ah[k], al[k], bh[0], bh[1], bl[0], bl[1]);
                        mma3(main[1], cross[1], ah[k], al[k], bh[2], bh[3], bl[2], bl[3]);
                    }
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            *(float2*)(to + 8 * i * TP + 16 * half + 8 * n) =
                                make_float2((main[n][2 * i] + cross[n][2 * i]) * down, (main[n][2 * i + 1] + cross[n][2 * i + 1]) * down);
                }
            };
            product(q_s, s.down * q_down, sum);
            if constexpr (MODE == DELTA) product(w_s, s.down * rec[Rec::SCALARS + W_DOWN], sum + SH::SUM_FLOATS);
        }
        // ---- the chunk's values as left operands (columns g, g + 8; tokens 16 k + 2 t4, + 1, + 8, + 9)
        float va[2][4][2];                                // [sixteen tokens][register][its two tokens]
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
                const float4 gg = *(const float4*)(rec + Rec::G + t);
                *(float4*)(u_s + j * TP + t) = make_float4(fmaf(-gg.x, y.x, v_s[t * VP + j]), fmaf(-gg.y, y.y, v_s[(t + 1) * VP + j]),
                                                           fmaf(-gg.z, y.z, v_s[(t + 2) * VP + j]), fmaf(-gg.w, y.w, v_s[(t + 3) * VP + j]));
                *(float4*)(z_s + j * TP + t) = make_float4(gg.x * z.x, gg.y * z.y, gg.z * z.z, gg.w * z.w);
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 x = *(const float2*)(u_s + (16 * cw + g + 8 * (i & 1)) * TP + 16 * k + 2 * t4 + 8 * (i >> 1));
                    va[k][i][0] = x.x; va[k][i][1] = x.y;
                }
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) va[k][i][e] = v_s[(16 * k + 2 * t4 + e + 8 * (i >> 1)) * VP + 16 * cw + g + 8 * (i & 1)];
        }
        unsigned largest = 0, largest_w = 0;
        float wf[2][4];                                   // w of the lane's tokens 16 k + 2 t4 (+ 1, + 8, + 9)
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) wf[k][i] = __shfl_sync(0xffffffffu, wt, 16 * k + 2 * t4 + (i & 1) + 8 * (i >> 1));
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    largest = max(largest, abs_bits(va[k][i][e]));
                    largest_w = max(largest_w, abs_bits(va[k][i][e] * wf[k][2 * (i >> 1) + e]));
                }
        largest = __reduce_max_sync(0xffffffffu, largest);
        largest_w = __reduce_max_sync(0xffffffffu, largest_w);
        lost |= max(largest, largest_w) >= 0x7f800000u;

        // ---- the state after the chunk
        {
            const Scale s = scale_of(largest_w);
            unsigned ah[2][4], al[2][4];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    split2(va[k][i][0] * wf[k][2 * (i >> 1)] * s.up, va[k][i][1] * wf[k][2 * (i >> 1) + 1] * s.up, ah[k][i], al[k][i]);
            const float down = s.down * k_down;
#pragma unroll
            for (int n = 0; n < NK; n += 2) {
                float main[2][4] = {}, cross[2][4] = {};
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int row = 16 * k + 8 * ((lane >> 3) & 1) + (lane & 7), col = KPW * kw + 8 * n + 8 * (lane >> 4);
                    unsigned bh[4], bl[4];
                    ldsm_t(bh, k_s + tile_at<DP>(row, col));
                    ldsm_t(bl, k_s + CT * DP + tile_at<DP>(row, col));
                    mma3(main[0], cross[0], ah[k], al[k], bh[0], bh[1], bl[0], bl[1]);
                    mma3(main[1], cross[1], ah[k], al[k], bh[2], bh[3], bl[2], bl[3]);
                }
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    float2 d = make_float2(decay, decay);
                    if constexpr (MODE == KEY_DECAY) d = *(const float2*)(rec + Rec::KEYS + KPW * kw + 8 * (n + m) + 2 * t4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) S[n + m][i] = fmaf((i & 1) ? d.y : d.x, S[n + m][i], (main[m][i] + cross[m][i]) * down);
                }
            }
        }
        // ---- P V of the tokens that the warp finishes
        float o[NT][4];
        if (KW <= 4 || kw < 4) {
            const Scale s = scale_of(largest);
            unsigned ah[2][4], al[2][4];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) split2(va[k][i][0] * s.up, va[k][i][1] * s.up, ah[k][i], al[k][i]);
            const float down = s.down * p_down;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float main[4] = {}, cross[4] = {};
                const int row = 8 * (NT * kw + n) + (lane & 7);
                unsigned bh[4], bl[4];                    // the four groups of eight tokens s
                ldsm(bh, p_s + score_at(row, 8 * (lane >> 3)));
                ldsm(bl, p_s + CT * CT + score_at(row, 8 * (lane >> 3)));
                mma3(main, cross, ah[0], al[0], bh[0], bh[1], bl[0], bl[1]);
                mma3(main, cross, ah[1], al[1], bh[2], bh[3], bl[2], bl[3]);
#pragma unroll
                for (int i = 0; i < 4; ++i) o[n][i] = (main[i] + cross[i]) * down;
            }
        }
        if constexpr (MODE == MATRIX_MEMORY) {            // q . n of the tokens: eight lanes a token, then n after the chunk
            const float* n_old = n_s + (c & 1) * DP;
            float* n_new = n_s + ((c + 1) & 1) * DP;
            float* nq_s = n_s + 2 * DP + (c & 1) * CT;
            for (int t = tid >> 3; t < CT; t += THREADS / 8) {
                float s = 0.f;
                for (int d = 8 * (lane & 7); d < DP; d += 64) {
                    const uint4 h4 = *(const uint4*)(q_s + tile_at<DP>(t, d)), l4 = *(const uint4*)(q_s + CT * DP + tile_at<DP>(t, d));
                    const __half2* h = reinterpret_cast<const __half2*>(&h4);
                    const __half2* l = reinterpret_cast<const __half2*>(&l4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 a = __half22float2(h[i]), b = __half22float2(l[i]), n = *(const float2*)(n_old + d + 2 * i);
                        s = fmaf(a.x + b.x, n.x, s);
                        s = fmaf(a.y + b.y, n.y, s);
                    }
                }
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                s += __shfl_xor_sync(0xffffffffu, s, 4);
                if ((lane & 7) == 0) nq_s[t] = s * q_down;
            }
            for (int d = tid; d < DP; d += THREADS) n_new[d] = fmaf(decay, n_old[d], w_more * rec[Rec::KEYS + d]);
        }
        if (p.stages > 2) copy_wait<1>(); else copy_wait<0>();       // the next chunk has landed
        float skipped[NT][4];
        if constexpr (MODE == HEAD_DECAY) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    skipped[n][i] = skip * v_s[(8 * (NT * kw + n) + 2 * t4 + (i & 1)) * VP + 16 * cw + g + (i >> 1) * 8];
        }
        const float row_sum = MODE == MATRIX_MEMORY ? rec[Rec::SUMS + lane] : 0.f;
        if constexpr (MODE != DELTA) {                    // the sums over the keys are complete, and this chunk's stage is free
            lost = __syncthreads_or(lost);
            if (lost) break;
        }
        float den_t = 1.f;
        if constexpr (MODE == MATRIX_MEMORY) {
            const float nq = p.out_scale * (gt * n_s[2 * DP + (c & 1) * CT + lane] + ht * row_sum);
            den_t = fmaxf(fabsf(nq), den) + 1e-6f;
        }
        if (KW <= 4 || kw < 4) {
            float* out = p.out + (size_t)tb * p.out_stride + (size_t)head * p.vdim + col0;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int t = 8 * (NT * kw + n) + 2 * t4, col = 16 * cw + g + 8 * r;
                    float2 z = make_float2(0.f, 0.f);
                    if constexpr (MODE == DELTA) z = *(const float2*)(extra + (COLS + col) * TP + t);
                    else {
#pragma unroll
                        for (int k = 0; k < KW; ++k) {
                            const float2 a = *(const float2*)(sum + (k * COLS + col) * TP + t);
                            z.x += a.x; z.y += a.y;
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float x;
                        if constexpr (MODE == DELTA) x = p.out_scale * ((e ? z.y : z.x) + o[n][2 * r + e]);
                        else {
                            x = p.out_scale * fmaf(__shfl_sync(0xffffffffu, gt, t + e), e ? z.y : z.x,
                                                   MODE == MATRIX_MEMORY ? __shfl_sync(0xffffffffu, ht, t + e) * o[n][2 * r + e] : o[n][2 * r + e]);
                            if constexpr (MODE == HEAD_DECAY) x += skipped[n][2 * r + e];
                            if constexpr (MODE == MATRIX_MEMORY) x /= __shfl_sync(0xffffffffu, den_t, t + e);
                        }
                        if (t + e < len && col < n_cols) out[(size_t)(t + e) * p.out_stride + col] = x;
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
int launch_walk(Walk p, cudaStream_t st) {
    using SH = Shape<KPW, KW, CW, MODE>;
    dim3 grid((p.vdim + SH::COLS - 1) / SH::COLS, p.heads, p.n_segments);
    // three stages where a multiprocessor holds one block anyway, two where two blocks then fit
    constexpr bool three = SH::bytes(3) <= 227 * 1024;
    p.stages = three && (long long)grid.x * grid.y * grid.z <= 148 ? 3 : 2;
    auto kernel = chunk_walk_kernel<KPW, KW, CW, MODE>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::bytes(three ? 3 : 2)) != cudaSuccess)
        return SPITE_LAUNCH_FAILED;
    // (in the ordinary way: started early, the blocks would sit on the multiprocessors of the kernel before, several to one)
    kernel<<<grid, SH::THREADS, SH::bytes(p.stages), st>>>(p);
    return spite_launch_status();
}

}  // namespace chunk
