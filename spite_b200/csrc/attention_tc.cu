// Attention over the paged cache for prompt portions on the fifth-generation tensor cores
// (bfloat16, head size 64 or 128, pages of a multiple of 64 keys, up to 128 query heads per kv head).
//
// A block owns two tiles of 128 rows of the score matrix: (token, query head of one kv group)
// pairs of consecutive tokens of one request, row = token * group + head; the second tile holds
// the tokens after the first's.  Both walk the same visible keys in tiles of 64 (one TMA box, never
// across a page), so a key or value tile is fetched once for 256 rows.  Roles:
//   warp 0     one lane loads the rows of q of both tiles once (three-dimensional TMA boxes: 64
//              elements x the group's heads x the tokens, which land row by row in the
//              128-byte-swizzled K-major layout) and then the K and V tiles into two rings of
//              four stages each;
//   warps 1-2  warp 1 allocates tensor memory (per row tile two score tiles of 64 columns and
//              the output tile of head-size columns); one lane of each issues, for its row
//              tile,  S = Q K^T  (128 x 64 x head size) and  O += P V  (128 x head size x 64; P
//              is read from tensor memory, V is used as it lies in the cache, as an MN-major
//              operand), two score tiles ahead of the softmax;
//   warps 3-10 four warps per row tile, one thread per row: read a score tile with tcgen05.ld,
//              scale and mask it, keep the running maximum and sum in float32, write P as
//              bfloat16 pairs over the first 32 columns of the score tile it came from
//              (tcgen05.st), and at the end divide the output by the sum.
// P never passes through shared memory: the tensor cores' operand reads from shared memory
// (q and the K tile for the scores, the V tile for the output) are what bounds the kernel, and P
// through shared memory would add a third to them.  A score tile's columns are written again
// (scores of the tile after next) only after the product that read P from them has completed.
// While one row tile's threads compute a softmax, the tensor cores work on the other tile's
// products.  (A kernel that allocates tensor memory gets one block per multiprocessor, so the
// overlap has to come from within the block.)  Blocks are persistent, one per multiprocessor:
// the work items (pair of row tiles, kv head) are dealt out round by round in alternating
// direction, heaviest first, or cut along the keys into equal shares (see Cut), and between items the
// block renews its barriers.
// The output accumulates in tensor memory.  A row's reference maximum moves only when the
// tile's maximum exceeds it by more than 8 (in log2 units): then the row's part of O and its
// sum are multiplied by 2^(old - new) before the next product is added.  P stays below 2^8, and
// the result is the same softmax(S) V up to rounding, since sum and output share the reference.
// A masked key has probability exactly 0, but 0 x (a value that is not a number) is not 0: the
// cache must hold finite values everywhere (it starts zeroed and only finite rows are appended).
//
// Score, mask and softmax: crates/spite-compute/src/flash_attn.rs:111-156; window rules in
// attention.cuh.  Every wait is bounded (see tcgen05.cuh); spite_attention_tc_error() returns
// and clears the code of a wait that gave up: 1 loader, 2 tensor-core issue, 3 softmax.
#include "attention.cuh"
#include "tcgen05.cuh"

namespace {
using namespace tc;

constexpr int BM = 128;                 // rows of one row tile
constexpr int BN = 64;                  // keys per tile (the softmax reads a score tile with one 64-column load)
constexpr int ST = 4;                   // stages of the K ring and of the V ring
constexpr int THREADS = 11 * 32;
constexpr int TMEM_COLS = 512;
constexpr int GROUP_COLS = 256;         // tensor-memory columns of one row tile: S0, S1 (64 each), O
constexpr float RESCALE_STEP = 8.f;     // log2 units
constexpr float LOG2E = 1.4426950408889634f;

__device__ int g_attn_tc_error = 0;
}  // namespace
// 1: the loader waited for a free stage, 2: the tensor-core issuer waited, 3: a softmax warp waited.
// (`extra_tx` is not used here.)
SPITE_WAIT_CONTROLS(attention_tc, g_attn_tc_error)
namespace {

// Work cut along the keys.  An item (pair of row tiles, kv head) costs its key tiles and CUT_ITEM more (to start and to end, about 7 us);
// the items laid end to end are one line, and every block takes an equal stretch of it.  What a stretch holds of an item that it shares
// with others is a part: its rows' output before the division, their maximum and their sum go to `partial`, and a kernel behind this one
// adds an item's parts up, in the order of the keys.
constexpr int CUT_PAIRS = 1024;         // most pairs of row tiles
constexpr int CUT_ITEM = 6;
constexpr int CUT_PIECE = 4;            // a part is no shorter than this many key tiles: a cut so close to an item's end moves there
constexpr int CUT_SHARE = 8;            // nor is a block's share
struct Cut {
    float* partial;                     // [blocks][2: a block's first part, its last][2 row tiles x (HD + 2) x 128], or null: items are not cut
    int4* items;                        // [blocks]: the item whose first cut is where block i begins (item, parts, first token, tokens); no parts: none
};

struct GroupBarriers {
    unsigned long long s_full[2], p_ready, pv_done, exp_done;
};
struct Barriers {
    unsigned long long q_full, k_full[ST], k_empty[ST], v_full[ST], v_empty[ST];
    GroupBarriers g[2];
    unsigned tmem_base;
    int abort_flag;
};

// 2^x by the special-function unit (relative error about 2^-22; 2^-inf = 0)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
template <int N> struct Count { static constexpr int value = N; };
typedef unsigned long long f2;                            // two packed floats
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
// The larger of two numbers, or NaN where one of them is NaN (fmaxf gives the other).
__device__ __forceinline__ float max_or_nan(float a, float b) {
    float v;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(v) : "f"(a), "f"(b));
    return v;
}
// 2^x for two numbers on the multiply-add units, x at most 127: x = n + f with n whole and |f| <= 1/2, a polynomial of degree 5 for 2^f
// (least worst relative error over [-1/2, 1/2], fitted by Lawson's iteration: 7.5e-8, 2.1e-7 with the roundings, as much as the
// special-function unit's) times 2^n.  As with the unit, NaN gives NaN, and what lies below -127 gives 0 (n = -127 makes the factor's
// bits all zero).  (n is not added to the polynomial's exponent, which would be one multiplication less: on a NaN's bits that gives a number.)
__device__ __forceinline__ void ex2_pair(f2 x, float& a, float& b) {
    auto both = [](float v) { return pack2(v, v); };
    float xa, xb;
    unpack2(x, xa, xb);
    x = pack2(max_or_nan(xa, -127.f), max_or_nan(xb, -127.f));
    const f2 n = add2(x, both(12582912.f));                // 1.5 * 2^23: n stands in the low bits
    const f2 f = fma2(add2(n, both(-12582912.f)), both(-1.f), x);
    f2 p = fma2(both(0.00132764445f), f, both(0.00967553724f));
    p = fma2(p, f, both(0.0555071346f));
    p = fma2(p, f, both(0.240221202f));
    p = fma2(p, f, both(0.693146944f));
    p = fma2(p, f, both(1.00000012f));
    float na, nb;
    unpack2(n, na, nb);
    const f2 two_n = pack2(__int_as_float((__float_as_int(na) << 23) + 0x3f800000), __int_as_float((__float_as_int(nb) << 23) + 0x3f800000));
    unpack2(mul2(p, two_n), a, b);
}
__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *(unsigned*)&v;
}

__host__ __device__ constexpr size_t slot_floats(int head_dim) { return 2 * (size_t)(head_dim + 2) * BM; }     // of a part

// What a row's output is multiplied by in the end: one over its sum, which the sink joins first; m is the row's reference in log2 units.
__device__ __forceinline__ float inverse_sum(const AttentionParams& p, int tok, int head, float m, float l) {
    float shrink = 1.f;
    if (p.has_sink) {                              // the sink's score in this kernel's units (powers of two)
        const float sink2 = sink_of(p, head) * LOG2E, m2 = fmaxf(m, sink2);
        shrink = (m == -INFINITY) ? 0.f : exp2f(m - m2);
        l = l * shrink + exp2f(sink2 - m2);
    }
    return shrink * gate_of(p, tok, head) / fmaxf(l, 1e-30f);
}

// NKB = head_dim / 64.  grid (blocks over (request, pair of token tiles), kv heads).
template <int NKB, int FORM>
__global__ void __launch_bounds__(THREADS, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const AttentionParams p, const StepTokens b,
               const PagedCache c, const AttnMmaExtra x, const int q_box_tokens, const int n_tile_pairs, const Cut cut,
               const WaitControl waits) {
    constexpr int HD = 64 * NKB;
    constexpr int Q_BYTES = NKB * BM * 128;              // q of one row tile
    constexpr int KT_BYTES = NKB * BN * 128;             // one K tile, one V tile
    extern __shared__ __align__(1024) unsigned char smem[];   // [Q0][Q1][K ring][V ring], each 1024-byte aligned
    __shared__ Barriers bars;
    __shared__ int line[CUT_PAIRS + 1];                       // what the pairs before cost (for one kv head)
    __shared__ __align__(16) float key_scales[FORM == FORM_ANY ? 8 : 1][BN];    // a softmax warp's copy of its tile's keys' factors
    pdl_wait();
    pdl_launch_dependents();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = p.num_heads, nkv = c.num_kv_heads, G = nq / nkv;
    const int tpt = x.tokens_per_block;                   // tokens of one row tile

    unsigned char* q_s = smem;
    unsigned char* k_s = q_s + 2 * Q_BYTES;
    unsigned char* v_s = k_s + ST * KT_BYTES;
    volatile int* abort_flag = &bars.abort_flag;
    int* const err_word = waits.error_word ? waits.error_word : &g_attn_tc_error;
    const long long wait_limit = waits.limit_cycles;

    auto init_barriers = [&](bool renew) {
        auto one = [&](unsigned long long* bar, unsigned count) {
            if (renew) mbar_inval(smem_u32(bar));
            mbar_init(smem_u32(bar), count);
        };
        one(&bars.q_full, 1);
        for (int s = 0; s < ST; ++s) {
            one(&bars.k_full[s], 1); one(&bars.k_empty[s], 2);     // both row tiles release a stage
            one(&bars.v_full[s], 1); one(&bars.v_empty[s], 2);
        }
        for (int g = 0; g < 2; ++g) {
            for (int s = 0; s < 2; ++s) one(&bars.g[g].s_full[s], 1);
            one(&bars.g[g].p_ready, 4);                            // one arrival per softmax warp
            one(&bars.g[g].pv_done, 1);
            one(&bars.g[g].exp_done, 4);
        }
        mbar_init_fence();
    };
    if (threadIdx.x == 0) {
        bars.abort_flag = 0;
        init_barriers(false);
    }
    if (warp == 1) tmem_alloc(&bars.tmem_base, TMEM_COLS);
    // The pair of row tiles `idx`: its request, first token, number of tokens (seg < 0: the caller counted more pairs than there are),
    // first key and key tiles, from the first key that its first token sees to its last token's own.
    struct Pair { int seg, t0, nt, k_begin, n_tiles; };
    auto pair_of = [&](int idx) {
        Pair r{-1, 0, 0, 0, 0};
        for (int s = 0; s < x.n_segments; ++s) {
            const int lo = x.cu_seqlens[s], n = x.cu_seqlens[s + 1] - lo;
            if (n < x.seg_min_tokens || n > x.seg_max_tokens) continue;   // another kernel serves this segment
            const int blocks = (n + 2 * tpt - 1) / (2 * tpt);
            if (idx < blocks) { r.seg = s; r.t0 = lo + idx * 2 * tpt; r.nt = min(2 * tpt, lo + n - r.t0); break; }
            idx -= blocks;
        }
        if (r.seg >= 0) {
            r.k_begin = (window_lowest(p.window_kind, p.window_size, b.positions[r.t0]) / BN) * BN;
            r.n_tiles = (b.positions[r.t0 + r.nt - 1] - r.k_begin) / BN + 1;
        }
        return r;
    };
    if (cut.partial)
        for (int j = threadIdx.x; j < n_tile_pairs; j += THREADS) {
            const int n = pair_of(n_tile_pairs - 1 - j).n_tiles;
            line[j + 1] = n ? n + CUT_ITEM : 0;
        }
    if (warp >= 3) {
        // rows of a q tile that the TMA box does not write: zero, so that their scores are plain numbers
        const int g = (warp - 3) >> 2, r = (warp & 3) * 32 + lane;
        if (r >= q_box_tokens * G) {
#pragma unroll
            for (int kb = 0; kb < NKB; ++kb)
#pragma unroll
                for (int ch = 0; ch < 8; ++ch)
                    *(uint4*)(q_s + g * Q_BYTES + kb * BM * 128 + r * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async();
    }
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = bars.tmem_base;

    // The line: item (pair n_tile_pairs - 1 - j, kv head h) begins at nkv * line[j] + h * its length.  Block i's stretch goes from cut i to
    // cut i + 1; cut i is at i equal shares, or at the item's start or end if it leaves less than CUT_PIECE key tiles on that side.
    long long line_end = 0, at = 0, stretch_end = 0;
    int sharers = 0;
    struct Place { int j, kvh, off, len; };
    auto place_of = [&](long long t) {                        // 0 <= t < line_end
        int lo = 0, hi = n_tile_pairs;                        // nkv * line[lo] <= t < nkv * line[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((long long)nkv * line[mid] <= t) lo = mid; else hi = mid;
        }
        const int len = line[lo + 1] - line[lo], rest = (int)(t - (long long)nkv * line[lo]);
        return Place{lo, rest / len, rest % len, len};
    };
    auto cut_at = [&](int i) {
        if (i >= sharers) return line_end;
        const long long t = line_end * i / sharers;
        if (t == 0) return t;
        const Place q = place_of(t);
        return q.off < CUT_ITEM + CUT_PIECE ? t - q.off : q.len - q.off < CUT_PIECE ? t + q.len - q.off : t;
    };
    if (cut.partial) {
        if (warp == 0) {
            int sum = 0;
            for (int j0 = 0; j0 < n_tile_pairs; j0 += 32) {
                int v = j0 + lane < n_tile_pairs ? line[j0 + lane + 1] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                if (j0 + lane < n_tile_pairs) line[j0 + lane + 1] = sum + v;
                sum += __shfl_sync(0xffffffffu, v, 31);
            }
            if (lane == 0) line[0] = 0;
        }
        __syncthreads();
        line_end = (long long)nkv * line[n_tile_pairs];
        sharers = (int)min((long long)gridDim.x, max(1ll, line_end / CUT_SHARE));
        if (line_end > 0 && blockIdx.x < sharers) { at = cut_at(blockIdx.x); stretch_end = cut_at(blockIdx.x + 1); }
        if (threadIdx.x == 0) {
            int4 mine = make_int4(0, 0, 0, 0);
            if (at < stretch_end) {
                const Place q = place_of(at);
                if (q.off > 0) {                              // the cuts within the item: those that leave CUT_PIECE tiles on either side
                    const long long t0 = at - q.off;
                    int first = -1, n = 0;
                    for (int i = (int)(t0 * sharers / line_end); i < sharers; ++i) {
                        const long long t = line_end * i / sharers;
                        if (t > t0 + q.len - CUT_PIECE) break;
                        if (i == 0 || t < t0 + CUT_ITEM + CUT_PIECE) continue;
                        if (n++ == 0) first = i;
                    }
                    if (first == blockIdx.x) {
                        const Pair r = pair_of(n_tile_pairs - 1 - q.j);
                        mine = make_int4(q.j * nkv + q.kvh, n + 1, r.t0, r.nt);
                    }
                }
            }
            cut.items[blockIdx.x] = mine;
        }
    }

    // Work items: (pair of row tiles of a request, kv head), numbered so that the work falls with the
    // number (later tokens see more keys).  Blocks are persistent.  Uncut, round r deals items r * blocks ..
    // (r + 1) * blocks - 1 to the blocks, in alternating direction, so that the shares come out alike.
    const int n_items = n_tile_pairs * nkv;
    for (int round = 0;; ++round) {
        int kvh, from = 0;
        bool part = false;
        Pair pair;
        if (cut.partial) {
            if (at >= stretch_end) break;
            const Place q = place_of(at);
            const int to = (int)min((long long)q.len, q.off + (stretch_end - at));
            kvh = q.kvh;
            at += to - q.off;
            from = max(0, q.off - CUT_ITEM);
            part = from > 0 || to < q.len;
            pair = pair_of(n_tile_pairs - 1 - q.j);
            pair.k_begin += from * BN;
            pair.n_tiles = to - CUT_ITEM - from;
        } else {
            const int item = round * gridDim.x + ((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
            if (item >= n_items) break;
            kvh = item % nkv;
            pair = pair_of(n_tile_pairs - 1 - item / nkv);
            if (pair.seg < 0) break;
        }
        const int seg = pair.seg, t0 = pair.t0, nt = pair.nt, k_begin = pair.k_begin, n_tiles = pair.n_tiles;
        const int* table = b.block_table + (size_t)seg * b.table_width;

        if (warp == 0) {
            if (lane == 0) {
                // ---- loader
                const unsigned q_bar = smem_u32(&bars.q_full);
                mbar_expect_tx(q_bar, (unsigned)(2 * NKB * q_box_tokens * G * 128));
#pragma unroll
                for (int g = 0; g < 2; ++g)
#pragma unroll
                    for (int kb = 0; kb < NKB; ++kb)
                        tma_load_3d(smem_u32(q_s + g * Q_BYTES + kb * BM * 128), &map_q, kb * 64, kvh * G, t0 + g * tpt, q_bar);
                int issued_k = 0, issued_v = 0;
                for (int i = 0; i < n_tiles; ++i) {
                    const int s = i % ST;
                    const unsigned ph = (i / ST) & 1;
                    const int j0 = k_begin + i * BN;
                    int page = table[j0 / c.page_size];
                    if (page < 0 || page >= c.n_pages) page = 0;   // a page behind every row's window: its keys are masked
                    const int y = (page * nkv + kvh) * c.page_size + j0 % c.page_size;
                    if (!mbar_wait(smem_u32(&bars.k_empty[s]), ph ^ 1, abort_flag, err_word, 1, wait_limit)) break;
                    mbar_expect_tx(smem_u32(&bars.k_full[s]), KT_BYTES);
#pragma unroll
                    for (int kb = 0; kb < NKB; ++kb)
                        tma_load_2d(smem_u32(k_s + s * KT_BYTES + kb * BN * 128), &map_k, kb * 64, y, smem_u32(&bars.k_full[s]));
                    ++issued_k;
                    if (!mbar_wait(smem_u32(&bars.v_empty[s]), ph ^ 1, abort_flag, err_word, 1, wait_limit)) break;
                    mbar_expect_tx(smem_u32(&bars.v_full[s]), KT_BYTES);
#pragma unroll
                    for (int kb = 0; kb < NKB; ++kb)
                        tma_load_2d(smem_u32(v_s + s * KT_BYTES + kb * BN * 128), &map_v, kb * 64, y, smem_u32(&bars.v_full[s]));
                    ++issued_v;
                }
                // the last releases of the stages must have arrived before the barriers are renewed for the next item
                for (int j = max(0, n_tiles - ST); j < n_tiles && !*abort_flag; ++j) {
                    if (!mbar_wait(smem_u32(&bars.k_empty[j % ST]), (j / ST) & 1, abort_flag, err_word, 1, wait_limit)) break;
                    if (!mbar_wait(smem_u32(&bars.v_empty[j % ST]), (j / ST) & 1, abort_flag, err_word, 1, wait_limit)) break;
                }
                if (*abort_flag) {
                    // copies in flight must land before the block gives its shared memory back
                    mbar_drain(q_bar, 0, wait_limit);
                    for (int j = max(0, issued_k - ST); j < issued_k; ++j) mbar_drain(smem_u32(&bars.k_full[j % ST]), (j / ST) & 1, wait_limit);
                    for (int j = max(0, issued_v - ST); j < issued_v; ++j) mbar_drain(smem_u32(&bars.v_full[j % ST]), (j / ST) & 1, wait_limit);
                }
            }
        } else {
            // ---- one of the two row tiles
            const int g = warp < 3 ? warp - 1 : (warp - 3) >> 2;
            GroupBarriers& gb = bars.g[g];
            const int tg0 = t0 + g * tpt;
            const int ntg = max(0, min(tpt, nt - g * tpt));
            // the key tiles from the first that a row tile's first token sees to its last token's own, [lo, hi] among the block's
            auto own_tiles = [&](int pos_first, int pos_last, int& lo, int& hi) {
                lo = max(0, window_lowest(p.window_kind, p.window_size, pos_first) / BN - k_begin / BN);
                hi = min(n_tiles, pos_last / BN - k_begin / BN + 1) - 1;
                if (hi < lo) { lo = 0; hi = -1; }
            };
            // this row tile's own; the second tile of a block may hold no token, and a part may hold none of a row tile's keys
            int first = 0, last = -1, p_first = 0, lo_last = 0;
            if (ntg > 0) {
                p_first = b.positions[tg0];
                const int p_last = b.positions[tg0 + ntg - 1];
                lo_last = window_lowest(p.window_kind, p.window_size, p_last);
                own_tiles(p_first, p_last, first, last);
            }
            const int n_own = last - first + 1;
            // the key tiles that both row tiles own, [shared_lo, shared_hi] among the block's: there the two take
            // turns at the exponentials
            int shared_lo = 0, shared_hi = -1;
            {
                const int og = g ^ 1, otg0 = t0 + og * tpt, ontg = max(0, min(tpt, nt - og * tpt));
                if (ontg > 0 && ntg > 0) {
                    const int op_first = b.positions[otg0], op_last = b.positions[otg0 + ontg - 1];
                    int olo, ohi;
                    own_tiles(op_first, op_last, olo, ohi);
                    shared_lo = max(first, olo);
                    shared_hi = min(last, ohi);
                }
            }
            const unsigned tmem_g = tmem + g * GROUP_COLS;
            unsigned char* q_g = q_s + g * Q_BYTES;

            if (warp < 3) {
                if (lane == 0) {
                    // ---- tensor-core issue for this row tile
                    const unsigned idesc_s = make_idesc(BM, BN), idesc_pv = make_idesc(BM, HD, true);
                    bool ok = mbar_wait(smem_u32(&bars.q_full), 0, abort_flag, err_word, 2, wait_limit);
                    // a key tile that this row tile does not need: wait until it has landed (so that the two
                    // row tiles never drift apart by more than the ring) and hand the stage back unread
                    auto pass_tile = [&](int i) {
                        const int s = i % ST;
                        const unsigned ph = (i / ST) & 1;
                        if (!mbar_wait(smem_u32(&bars.k_full[s]), ph, abort_flag, err_word, 2, wait_limit)) return false;
                        mbar_arrive(smem_u32(&bars.k_empty[s]));
                        if (!mbar_wait(smem_u32(&bars.v_full[s]), ph, abort_flag, err_word, 2, wait_limit)) return false;
                        mbar_arrive(smem_u32(&bars.v_empty[s]));
                        return true;
                    };
                    // scores of own tile li (key tile first + li) into score buffer li & 1, whose columns held
                    // P of tile li - 2: the product that read it must have completed
                    auto issue_scores = [&](int li) {
                        const int i = first + li, s = i % ST, sb = li & 1;
                        if (!mbar_wait(smem_u32(&bars.k_full[s]), (i / ST) & 1, abort_flag, err_word, 2, wait_limit)) return false;
                        if (li >= 2 && !mbar_wait(smem_u32(&gb.pv_done), li & 1, abort_flag, err_word, 2, wait_limit)) return false;
                        fence_after();
                        const unsigned qa = smem_u32(q_g), ka = smem_u32(k_s + s * KT_BYTES);
#pragma unroll
                        for (int ks = 0; ks < HD / 16; ++ks)
                            mma(tmem_g + sb * BN, smem_desc_k_major(qa + (ks / 4) * BM * 128 + (ks % 4) * 32),
                                smem_desc_k_major(ka + (ks / 4) * BN * 128 + (ks % 4) * 32), idesc_s, ks > 0 ? 1u : 0u);
                        commit(smem_u32(&gb.s_full[sb]));
                        commit(smem_u32(&bars.k_empty[s]));
                        return true;
                    };
                    for (int i = 0; i < first && ok; ++i) ok = pass_tile(i);
                    if (ok && n_own > 0) ok = issue_scores(0);
                    if (ok && n_own > 1) ok = issue_scores(1);
                    for (int li = 0; li < n_own && ok; ++li) {
                        const int i = first + li, s = i % ST;
                        ok = mbar_wait(smem_u32(&gb.p_ready), li & 1, abort_flag, err_word, 2, wait_limit) &&
                             mbar_wait(smem_u32(&bars.v_full[s]), (i / ST) & 1, abort_flag, err_word, 2, wait_limit);
                        if (!ok) break;
                        fence_after();
                        const unsigned va = smem_u32(v_s + s * KT_BYTES);
#pragma unroll
                        for (int ks = 0; ks < BN / 16; ++ks)
                            mma_a_tmem(tmem_g + 2 * BN, tmem_g + (li & 1) * BN + ks * 8, smem_desc(va + ks * 16 * 128, BN * 128, 1024),
                                       idesc_pv, (li > 0 || ks > 0) ? 1u : 0u);
                        commit(smem_u32(&gb.pv_done));
                        commit(smem_u32(&bars.v_empty[s]));
                        if (li + 2 < n_own) ok = issue_scores(li + 2);
                    }
                    for (int i = last + 1; i < n_tiles && ok; ++i) ok = pass_tile(i);
                }
            } else {
                // ---- softmax: one thread per row; warp w may read tensor-memory lanes [32 (w % 4), + 32)
                const int quarter = warp & 3;
                const int r = quarter * 32 + lane;
                const bool row_ok = r < ntg * G;
                const int tok = tg0 + (row_ok ? r / G : 0), head = kvh * G + (row_ok ? r % G : 0);
                const int pos = row_ok ? b.positions[tok] : -1;   // a row without a token sees no key
                const int lo = window_lowest(p.window_kind, p.window_size, max(pos, 0));
                const float scale = p.softmax_scale * LOG2E;
                // a bias that grows with the distance to the key, in units of the raw scores (they are multiplied by
                // the scale afterwards): its rounding error is relative to the bias itself
                const bool biased = p.head_slopes != nullptr;
                const float bias_raw = slope_of(p, head) / p.softmax_scale;
                // a cap on the scaled scores, in units of the raw ones; the argument of 2^x that gives e^(2 s scale / cap)
                const float cap_raw = p.score_softcap > 0.f ? p.score_softcap / p.softmax_scale : 0.f;
                const float cap_arg = p.score_softcap > 0.f ? 2.f * LOG2E * p.softmax_scale / p.score_softcap : 0.f;
                const float inv_cap_raw = p.score_softcap > 0.f ? p.softmax_scale / p.score_softcap : 0.f;
                // a number per distance, brought into the units of the raw scores as it is added
                const float* dist_row = FORM == FORM_ANY ? distance_row_of(p, head) : nullptr;
                const float per_scale = 1.f / p.softmax_scale;
                // the keys' factors: a lane asks for two of the next tile's while this tile is worked on
                const bool scaled = FORM == FORM_ANY && c.key_scale != nullptr;
                float* const scale_s = key_scales[FORM == FORM_ANY ? warp - 3 : 0];
                float2 next_scale = make_float2(1.f, 1.f);
                auto ask_scales = [&](int li) {
                    if (!scaled || li >= n_own) return;
                    const int j = k_begin + (first + li) * BN;
                    int page = table[j / c.page_size];
                    if (page < 0 || page >= c.n_pages) page = 0;        // (as the loader: behind every row's window)
                    next_scale = *(const float2*)(key_scale_of(c, page, kvh, j) + 2 * lane);
                };
                ask_scales(0);
                const unsigned lane_base = tmem_g + ((unsigned)(quarter * 32) << 16);
                float m_ref = -INFINITY, l = 0.f;
                bool ok = true;
                for (int li = 0; li < n_own; ++li) {
                    const int sb = li & 1;
                    if (scaled) {
                        __syncwarp();                                   // every lane has read the tile before's
                        *(float2*)(scale_s + 2 * lane) = next_scale;
                        __syncwarp();
                        ask_scales(li + 1);
                    }
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&gb.s_full[sb]), (li >> 1) & 1, abort_flag, err_word, 3, wait_limit));
                    if (!ok) break;
                    fence_after();
                    float s[BN];
                    ld64(s, lane_base + sb * BN);
                    const int j0 = k_begin + (first + li) * BN;
                    const bool open = j0 >= lo_last && j0 + BN - 1 <= p_first;   // every key visible to every row with a token
                    // maximum of the raw scores (the scale is positive); four running values shorten the chain
                    float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                    // The bias of key j0 + e is bias_raw * (j0 - pos) + bias_raw * e: the second term is one multiply-add an
                    // element with a constant that the compiler knows; the first is the same for the whole tile and joins
                    // the maximum and the exponent's offset below.
                    float tile_bias = biased ? bias_raw * (float)(j0 - pos) : 0.f;
                    if (scaled) {
#pragma unroll
                        for (int e = 0; e < BN; e += 4) {
                            const ulonglong2 f = *(const ulonglong2*)(scale_s + e);
                            unpack2(mul2(pack2(s[e], s[e + 1]), f.x), s[e], s[e + 1]);
                            unpack2(mul2(pack2(s[e + 2], s[e + 3]), f.y), s[e + 2], s[e + 3]);
                        }
                    }
                    if (FORM == FORM_CAP || (FORM == FORM_ANY && cap_raw > 0.f)) {
                        // cap tanh(s scale / cap) in units of the raw scores: where every score of the warp's rows is small against
                        // the cap the series (multiply-adds, two scores an instruction), else 1 - 2 / (e^(2x) + 1), whose two
                        // special-function operations a score would bind the kernel; the errors are far below a bfloat16 weight's
                        float big[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int e = 0; e < BN; ++e) big[e & 3] = fmaxf(big[e & 3], fabsf(s[e]));
                        if (__all_sync(0xffffffffu, fmaxf(fmaxf(big[0], big[1]), fmaxf(big[2], big[3])) <= CAP_SERIES * cap_raw)) {
                            const f2 inv = pack2(inv_cap_raw, inv_cap_raw), one = pack2(1.f, 1.f), c1 = pack2(CAP_C1, CAP_C1),
                                     c2 = pack2(CAP_C2, CAP_C2), c3 = pack2(CAP_C3, CAP_C3), c4 = pack2(CAP_C4, CAP_C4), c5 = pack2(CAP_C5, CAP_C5);
#pragma unroll
                            for (int e = 0; e < BN; e += 2) {
                                const f2 v = pack2(s[e], s[e + 1]), t = mul2(v, inv), y = mul2(t, t);
                                unpack2(mul2(v, fma2(y, fma2(y, fma2(y, fma2(y, fma2(y, c5, c4), c3), c2), c1), one)), s[e], s[e + 1]);
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < BN; ++e)
                                s[e] = fmaf(-2.f * cap_raw, reciprocal_approx(ex2(s[e] * cap_arg) + 1.f), cap_raw);
                        }
                    }
                    if (biased) {
#pragma unroll
                        for (int e = 0; e < BN; ++e) s[e] = fmaf(bias_raw, (float)e, s[e]);
                    }
                    if (FORM == FORM_ANY && dist_row) {
                        // The numbers change with the distance near the query and hardly further away: where every row of the
                        // warp has one number for its whole tile, that joins the tile's common term; else each key's is read
                        // (a row's distances lie side by side, the repeated ends take the tile's overhang).
                        const int n = pos - j0, len1 = p.distance_len - 1;       // the distance of the tile's first key
                        const int n_hi = max(min(n, len1), 0), n_lo = max(min(n - BN + 1, len1), 0);
                        if (__all_sync(0xffffffffu, p.distance_runs[n_hi] <= n_lo)) {
                            tile_bias = fmaf(dist_row[n_lo], per_scale, tile_bias);
                        } else {
                            const float* d = dist_row + min(max(n, -1), len1 + SPITE_DISTANCE_PAD);
#pragma unroll
                            for (int e = 0; e < BN; ++e) s[e] = fmaf(d[-e], per_scale, s[e]);
                        }
                    }
                    if (!open) {                                   // a tile on a window's edge or on the diagonal
#pragma unroll
                        for (int e = 0; e < BN; ++e) {
                            const int j = j0 + e;
                            s[e] = (j >= lo && j <= pos) ? s[e] : -INFINITY;
                        }
                    }
#pragma unroll
                    for (int e = 0; e < BN; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], s[e]);
                    const float mx = (fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) + tile_bias) * scale;
                    const bool need = mx > m_ref + RESCALE_STEP;
                    float corr = 1.f;
                    if (need) { corr = exp2f(m_ref - mx); l *= corr; m_ref = mx; }
                    const float neg_m = (m_ref == -INFINITY) ? 0.f : fmaf(tile_bias, scale, -m_ref);
                    // Over the key tiles that both own, the two row tiles take turns at the exponentials (key tile i
                    // of the first row tile, key tile i of the second, key tile i + 1 of the first, ...): the
                    // special-function units serve one at full rate while the tensor cores work for the other,
                    // instead of both halves of the block computing and then both waiting.  Both count their
                    // turns from the first shared key tile, so each is at most one phase behind the other's barrier.
                    const int turn = first + li - shared_lo;
                    const bool takes_turns = turn >= 0 && first + li <= shared_hi;
                    if (takes_turns && (g == 1 || turn > 0)) {
                        const int before = g == 0 ? turn - 1 : turn;      // the other row tile's turn before this one
                        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.g[g ^ 1].exp_done), before & 1, abort_flag, err_word, 3, wait_limit));
                        if (!ok) break;
                    }
                    // Three of sixteen pairs go through the multiply-add units instead (not on a window's edge or the diagonal, where a
                    // masked key must get 0), and the turn is passed on a quarter before the end, so that the other row tile's first
                    // exponentials follow the last ones here.  us, the kernel alone in a loop, cut, 2,048 tokens behind 6,144, 40 heads: 343; turn
                    // passed early 336; one pair in 4 317; both 310; 3 in 16 307; one pair in 2, 3 328, 327; without turns 324.  (A polynomial that
                    // passed over NaN; with the one above 1.3 % more.  With L2 flushed between the calls 320 and 325.)
                    unsigned packed[BN / 2];
                    f2 sum2[4] = {0ull, 0ull, 0ull, 0ull};
                    const f2 scale2 = pack2(scale, scale), neg_m2 = pack2(neg_m, neg_m);
                    auto weights = [&](auto mixed) {
#pragma unroll
                        for (int e = 0; e < BN; e += 2) {
                            if (e == BN * 3 / 4) {
                                __syncwarp();
                                if (takes_turns && lane == 0) mbar_arrive(smem_u32(&gb.exp_done));
                            }
                            const f2 x = fma2(pack2(s[e], s[e + 1]), scale2, neg_m2);
                            float a, bb;
                            if (decltype(mixed)::value && ((e / 2) % 16 == 3 || (e / 2) % 16 == 8 || (e / 2) % 16 == 13)) {
                                ex2_pair(x, a, bb);
                            } else {
                                unpack2(x, a, bb);
                                a = ex2(a);
                                bb = ex2(bb);
                            }
                            sum2[(e >> 1) & 3] = add2(sum2[(e >> 1) & 3], pack2(a, bb));
                            packed[e / 2] = pack_bf16(a, bb);
                        }
                    };
                    if (open) weights(Count<1>{}); else weights(Count<0>{});
                    const f2 sums = add2(add2(sum2[0], sum2[1]), add2(sum2[2], sum2[3]));
                    float sum_a, sum_b;
                    unpack2(sums, sum_a, sum_b);
                    const float sum = sum_a + sum_b;
                    l += sum;
                    if (li > 0) {
                        // The product of the tile before must have left O before its rows are rescaled.  The wait is
                        // made for every tile, needed or not: a wait by parity is only right while the waiter is
                        // at most one phase behind the barrier.
                        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&gb.pv_done), (li - 1) & 1, abort_flag, err_word, 3, wait_limit));
                        if (!ok) break;
                        if (__any_sync(0xffffffffu, need)) {
                            fence_after();
#pragma unroll 1
                            for (int c0 = 0; c0 < HD; c0 += 32) {
                                float o[32];
                                ld32(o, lane_base + 2 * BN + c0);
#pragma unroll
                                for (int e = 0; e < 32; ++e) o[e] *= corr;
                                st32(lane_base + 2 * BN + c0, o);
                            }
                        }
                    }
                    st32(lane_base + sb * BN, packed);              // P over the first half of the score tile just read
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&gb.p_ready));
                }
                if (ok && n_own > 0)
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&gb.pv_done), (n_own - 1) & 1, abort_flag, err_word, 3, wait_limit));
                if (ok && n_own > 0) {
                    fence_after();
                    const float inv = part ? 0.f : inverse_sum(p, tok, head, m_ref, l);
                    __nv_bfloat16* dst = (__nv_bfloat16*)p.out + out_row_of(p, tok, head) * HD;
                    float* to = cut.partial + (size_t)(2 * blockIdx.x + (from == 0)) * slot_floats(HD) + g * HD * BM + r;
#pragma unroll 1
                    for (int c0 = 0; c0 < HD; c0 += 32) {
                        float o[32];
                        ld32(o, lane_base + 2 * BN + c0);          // warp-collective: every lane takes part
                        if (!row_ok) continue;
                        if (part) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) __stcg(to + (c0 + e) * BM, o[e]);    // a column's rows side by side
                            continue;
                        }
#pragma unroll
                        for (int e = 0; e < 32; e += 8)
                            *(uint4*)(dst + c0 + e) = make_uint4(pack_bf16(o[e] * inv, o[e + 1] * inv), pack_bf16(o[e + 2] * inv, o[e + 3] * inv),
                                                                 pack_bf16(o[e + 4] * inv, o[e + 5] * inv), pack_bf16(o[e + 6] * inv, o[e + 7] * inv));
                    }
                }
                if (part)
                    __stcg((float2*)(cut.partial + (size_t)(2 * blockIdx.x + (from == 0)) * slot_floats(HD) + 2 * HD * BM) + g * BM + r,
                           make_float2(n_own > 0 ? m_ref : -INFINITY, n_own > 0 ? l : 0.f));
            }
        }
        // end of the item: everything asynchronous has been waited for; renew the barriers
        fence_before();
        __syncthreads();
        fence_after();
        if (*abort_flag) break;
        if (threadIdx.x == 0) init_barriers(true);
        __syncthreads();
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_free(tmem, TMEM_COLS);
    }
}

// Adds up the parts of the items that were cut.  grid (cuts, head_dim / JOIN_COLS), a thread a row; part 0 of an item is the last of the
// block before its first cut, part k the first of the block behind its cut k.
constexpr int JOIN_COLS = 16;                                 // a thread's elements of a row
__global__ void __launch_bounds__(2 * BM) attn_tc_join_kernel(const AttentionParams p, const Cut cut, int nkv, int tpt, int hd) {
    pdl_wait();
    pdl_launch_dependents();
    const int4 item = __ldcg(cut.items + blockIdx.x);
    if (item.y < 2) return;
    const int G = p.num_heads / nkv, g = threadIdx.x / BM, r = threadIdx.x % BM, c0 = blockIdx.y * JOIN_COLS;
    if (r >= min(tpt, item.w - g * tpt) * G) return;
    const int tok = item.z + g * tpt + r / G, head = (item.x % nkv) * G + r % G;
    auto slot = [&](int k) { return cut.partial + (2 * (size_t)blockIdx.x + 2 * k - (k ? 2 : 1)) * slot_floats(hd); };
    float m = -INFINITY, l = 0.f, o[JOIN_COLS];
#pragma unroll
    for (int e = 0; e < JOIN_COLS; ++e) o[e] = 0.f;
    // N parts from part k0 on: their loads are asked for together
    auto add = [&](auto n, int k0) {
        constexpr int N = decltype(n)::value;
        float2 ml[N];
        float v[N][JOIN_COLS];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float* from = slot(min(k0 + k, item.y - 1));
            ml[k] = __ldcg((const float2*)(from + 2 * hd * BM) + threadIdx.x);
#pragma unroll
            for (int e = 0; e < JOIN_COLS; ++e) v[k][e] = __ldcg(from + (size_t)(g * hd + c0 + e) * BM + r);
        }
        float top = m;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (k0 + k >= item.y) ml[k].x = -INFINITY;
            top = fmaxf(top, ml[k].x);
        }
        const float keep = m == -INFINITY ? 0.f : exp2f(m - top);
        m = top;
        l *= keep;
#pragma unroll
        for (int e = 0; e < JOIN_COLS; ++e) o[e] *= keep;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (ml[k].x == -INFINITY) continue;               // (a part without a key for this row has left nothing there)
            const float w = exp2f(ml[k].x - m);
            l = fmaf(w, ml[k].y, l);
#pragma unroll
            for (int e = 0; e < JOIN_COLS; ++e) o[e] = fmaf(w, v[k][e], o[e]);
        }
    };
    if (item.y == 2) add(Count<2>{}, 0);
    else for (int k0 = 0; k0 < item.y; k0 += 4) add(Count<4>{}, k0);
    const float inv = inverse_sum(p, tok, head, m, l);
    __nv_bfloat16* dst = (__nv_bfloat16*)p.out + out_row_of(p, tok, head) * hd + c0;
#pragma unroll
    for (int e = 0; e < JOIN_COLS; e += 8)
        *(uint4*)(dst + e) = make_uint4(pack_bf16(o[e] * inv, o[e + 1] * inv), pack_bf16(o[e + 2] * inv, o[e + 3] * inv),
                                        pack_bf16(o[e + 4] * inv, o[e + 5] * inv), pack_bf16(o[e + 6] * inv, o[e + 7] * inv));
}

template <int NKB>
int launch(const AttentionParams& p, const StepTokens& b, const PagedCache& c, const AttnMmaExtra& x, int n_blocks,
           int n_sm, const Cut& cut, cudaStream_t st) {
    const int hd = 64 * NKB, nq = p.num_heads, nkv = c.num_kv_heads, G = nq / nkv;
    const int box_tokens = x.tokens_per_block < b.n_tokens ? x.tokens_per_block : b.n_tokens;
    CUtensorMap mq, mk, mv;
    {
        cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)nq, (cuuint64_t)b.n_tokens};
        cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)nq * hd * 2};
        cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)box_tokens};
        if (!make_map(&mq, p.q, 3, dims, strides, box)) return SPITE_LAUNCH_FAILED;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)hd, (cuuint64_t)c.n_pages * nkv * c.page_size};
        cuuint64_t strides[1] = {(cuuint64_t)hd * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)BN};
        if (!make_map(&mk, c.kv, 2, dims, strides, box)) return SPITE_LAUNCH_FAILED;
        if (!make_map(&mv, (const __nv_bfloat16*)c.kv + c.v_offset, 2, dims, strides, box)) return SPITE_LAUNCH_FAILED;
    }
    const size_t smem = 2 * (size_t)NKB * BM * 128 + 2 * ST * (size_t)NKB * BN * 128;
    const int form = score_form_of(p, c);
    auto k = form == FORM_ANY ? attn_tc_kernel<NKB, FORM_ANY> : form == FORM_CAP ? attn_tc_kernel<NKB, FORM_CAP> : attn_tc_kernel<NKB, FORM_PLAIN>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return SPITE_LAUNCH_FAILED;
    const long long items = (long long)n_blocks * nkv;
    const int grid = (int)(items < n_sm && !cut.partial ? items : n_sm);
    SPITE_LAUNCH(k, grid, THREADS, smem, st, mq, mk, mv, p, b, c, x, box_tokens, n_blocks, cut, s_waits);
    if (cut.partial) SPITE_LAUNCH(attn_tc_join_kernel, dim3(grid, hd / JOIN_COLS), 2 * BM, 0, st, p, cut, nkv, x.tokens_per_block, hd);
    return spite_launch_status();
}

// 2^x of pairs, for tests of ex2_pair
__global__ void ex2_pairs_kernel(const float2* x, float2* y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ex2_pair(pack2(x[i].x, x[i].y), y[i].x, y[i].y);
}

}  // namespace

// y = 2^x for n_pairs pairs of floats as the attention's weights in unmasked key tiles are made
SPITE_API int spite_attention_exp2_pairs(const float* x, float* y, int n_pairs, void* stream) {
    if (!x || !y || n_pairs < 0) return SPITE_BAD_ARG;
    if (((uintptr_t)x | (uintptr_t)y) & 7) return SPITE_UNSUPPORTED;
    if (n_pairs == 0) return SPITE_OK;
    ex2_pairs_kernel<<<(n_pairs - 1) / 256 + 1, 256, 0, (cudaStream_t)stream>>>((const float2*)x, (float2*)y, n_pairs);
    return spite_launch_status();
}

static int paged_attention_tc(const AttentionParams* p, const StepTokens* b, const PagedCache* c, const AttnMmaExtra* x, int n_blocks, int n_sm,
                              const Cut& cut, void* stream) {
    if (n_sm < 1) return SPITE_BAD_ARG;
    if (!p || !b || !c || !x || !p->q || !p->out || !x->cu_seqlens || !c->kv) return SPITE_BAD_ARG;
    if (!b->positions || !b->block_table || b->n_tokens < 0 || b->table_width < 1) return SPITE_BAD_ARG;
    if (p->num_heads < 1 || c->num_kv_heads < 1 || p->num_heads % c->num_kv_heads) return SPITE_BAD_ARG;
    if (p->window_kind < 0 || p->window_kind > 2) return SPITE_BAD_ARG;
    if (p->window_kind != SPITE_WINDOW_FULL && p->window_size < 1) return SPITE_BAD_ARG;
    if (!distance_bias_ok(p)) return SPITE_BAD_ARG;
    if (x->n_segments < 1 || x->tokens_per_block < 1 || n_blocks < 0 || c->n_pages < 1 || c->page_size < 1) return SPITE_BAD_ARG;
    const int G = p->num_heads / c->num_kv_heads;
    if ((c->head_dim != 64 && c->head_dim != 128) || G > BM || c->page_size % BN) return SPITE_UNSUPPORTED;
    if (x->tokens_per_block * G > BM) return SPITE_BAD_ARG;
    if ((long long)n_blocks * c->num_kv_heads > 0x7fffffffll || p->num_heads > 256 * c->num_kv_heads) return SPITE_UNSUPPORTED;
    if ((long long)c->n_pages * c->num_kv_heads * c->page_size > 0x7fffffffll) return SPITE_UNSUPPORTED;   // TMA coordinates are int32
    if ((((uintptr_t)p->q | (uintptr_t)p->out | (uintptr_t)c->kv | (uintptr_t)c->key_scale) & 15) || (c->v_offset & 7)) return SPITE_UNSUPPORTED;
    if (b->n_tokens == 0 || n_blocks == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    return c->head_dim == 64 ? launch<1>(*p, *b, *c, *x, n_blocks, n_sm, cut, st) : launch<2>(*p, *b, *c, *x, n_blocks, n_sm, cut, st);
}

// `tokens_per_block`: tokens of one row tile, tokens_per_block * (query heads per kv head) <= 128; a block
// serves two row tiles.  `n_blocks` = sum over the served segments of ceil(tokens / (2 tokens_per_block)),
// computed by the caller; `n_sm`: number of multiprocessors (one persistent block each).
SPITE_API int spite_paged_attention_tc(const AttentionParams* p, const StepTokens* b, const PagedCache* c,
                                       const AttnMmaExtra* x, int n_blocks, int n_sm, void* stream) {
    return paged_attention_tc(p, b, c, x, n_blocks, n_sm, Cut{nullptr, nullptr}, stream);
}

// The same with the work cut along the keys into n_sm equal shares, and a second kernel that adds the parts up.  `scratch`: n_sm * (4 * (head_dim +
// 2) * 128 + 4) floats.
SPITE_API int spite_paged_attention_tc_cut(const AttentionParams* p, const StepTokens* b, const PagedCache* c,
                                           const AttnMmaExtra* x, int n_blocks, int n_sm, float* scratch, long long n_floats, void* stream) {
    if (!scratch || n_sm < 1 || !c || c->head_dim < 1) return SPITE_BAD_ARG;
    const long long slots = 2ll * n_sm * (long long)slot_floats(c->head_dim);
    if (n_blocks > CUT_PAIRS || ((uintptr_t)scratch & 15) || slots + 4ll * n_sm > n_floats) return SPITE_UNSUPPORTED;
    return paged_attention_tc(p, b, c, x, n_blocks, n_sm, Cut{scratch, (int4*)(scratch + slots)}, stream);
}
