// Recurrent mixers whose state is a matrix per head that decays and takes one outer product a token, carried from token to
// token in float32 in the request's state slot.  One walk serves three designs:
//
//   state space (Mamba-2):   dt = softplus(a + dt_bias),  S <- exp(-exp(A_log) dt) S + dt k v^T,   o = S^T q + D v
//                            (one decay a head and token; q and k shared by a group of heads; read after the write)
//   decaying memory (RWKV):  o = S^T q + (sum_i q_i u_i k_i) v,   S <- diag(w) S + k v^T,   w = exp(-exp(z + w0))
//                            (a decay per key channel; the token itself enters the read-out through the bonus u)
//   gated linear attention:  S <- diag(w) S + k v^T,   o = c S^T q,   w = sigmoid(z)^(1/tau),   z = A_2 a + b
//                            (a decay per key channel from a short vector a; read after the write)
//
// S is [dim keys, vdim values], zeros at the start of a sequence.  Everything is float32.
//
// Unlike a delta rule, what a token writes does not depend on the state, so the walk is bound by what its warps can issue,
// not by one token's chain.  A warp is LR lanes along the keys times 32 / LR lanes along the values; a lane holds 4 RPV
// key rows (as packed pairs, for the two-at-a-time multiply-adds of sm_100) of CC value columns.  TB tokens form a batch:
// one more warp of the block brings their inputs into one stage of a shared-memory ring by asynchronous copies three batches
// ahead (so that the walking warps spend nothing on it; its lanes keep the addresses of what they copy in registers), one barrier stands between two batches, and the batch's TB * CC
// partial read-outs a lane are summed over the LR lanes by a halving exchange that leaves every lane TB * CC / LR finished
// numbers.  The order of the sums depends on the head's sizes alone, so the result does not depend on how a sequence was
// cut into steps.
//
// The slot holds S transposed: value column j's keys are contiguous, [vdim, dim4] with dim4 = dim rounded up to a multiple
// of four (the padding stays zero), so that a lane's rows are whole 16-byte groups and a warp's loads whole lines.
//
// Prompts and their portions go 32 tokens at a time on the tensor cores (chunk.cuh), for up to 128 keys.  With b_t the sum of a chunk's
// log decays up to token t: the scores P[t, s] = (q_t . k_s) e^(b_t - b_s) dt_s (s <= t) where one number a head decays, and
// sum_i q_ti k_si e^(b_ti - b_si) where every key channel does; the operands Q, K of the second kind carry e^(b_t) and e^(b_last - b_s).
// No exponent is ever positive.  The kernels below make these for all chunks and heads of a step at once.
#include "chunk.cuh"

SPITE_WAIT_CONTROLS(scan, chunk::walk_error)

struct ScanParams {
    const float* q; const float* k; const float* v;       // first element of token 0's q, k [kv_heads * dim], v [heads * vdim]
    long long q_stride, k_stride, v_stride;               // floats between two tokens' rows
    const float* w; long long w_stride;                   // decay per key channel [tokens, heads * dim], or null: per head
    const float* scalars;                                 // [tokens, heads, 4]: (decay, dt, -, -) without w; (bonus, -, -, -) with w;
                                                          // not read (null) by gated linear attention
    const float* skip;                                    // [heads] the factor D on v in the read-out, or null
    float* out; long long out_stride;                     // [tokens, heads * vdim]
    float* state; long long slot_stride;                  // state + slot * slot_stride + head * vdim * dim4
    const int* cu_seqlens; const int* slots;
    int n_segments, n_tokens, heads, kv_heads, dim, vdim;
    float out_scale;                                      // gated linear attention: the factor c on the read-out
    int n_long;                                           // the walks in chunks: how many segments they take, if that is known
};

namespace {

using namespace chunk;

typedef unsigned long long f2;                            // two packed floats

__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

constexpr int RING = 4;

constexpr int MAX_WARPS = 4;                              // walking warps a block

// the three designs
enum Walk { PER_HEAD = 0, PER_CHANNEL_BONUS = 1, PER_CHANNEL = 2 };

template <int LR, int RPV, int CC, int TB, int WALK>
struct WalkShape {
    static constexpr bool CH = WALK != PER_HEAD;          // a decay per key channel
    static constexpr bool SCALARS = WALK != PER_CHANNEL;  // a token brings scalars
    static constexpr int DP = LR * RPV * 4;               // key rows a warp covers
    static constexpr int WC = 32 / LR * CC;               // value columns a warp covers
    static constexpr int ROWS = CH ? 3 : 2;               // q, k (and w) of a token
    static constexpr int TOKEN = ROWS * DP + WC * MAX_WARPS + 4;      // floats of a token's stage
    static constexpr int KEEP = TB * CC / LR;             // finished numbers a lane
    static_assert(KEEP >= 1 && KEEP * LR == TB * CC && TOKEN % 4 == 0, "a batch's read-outs must fill the lanes");
};

// All threads of the block (the number is a multiple of 32).
__device__ __forceinline__ void block_barrier(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

// What one lane of the bringing warp copies of every token, in 16-byte groups (rows that are whole groups).
template <typename SH, int TB>
struct Bringer {
    static constexpr bool CH = SH::ROWS == 3;
    static constexpr int V = SH::ROWS * SH::DP;
    static constexpr int SLOTS = (SH::ROWS * (SH::DP / 4) + SH::WC * MAX_WARPS / 4 + 1 + 31) / 32;
    const float* src[SLOTS];
    long long stride[SLOTS];
    int dst[SLOTS];                                       // floats into a token's stage; < 0: nothing

    __device__ __forceinline__ Bringer(const ScanParams& p, const float* qp, const float* kp, const float* wp, const float* vp,
                                       const float* sp, int n_cols, long long t0, int lane) {
        const int du = p.dim >> 2, vu = n_cols >> 2, rows = SH::ROWS * du;
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            const int e = lane + 32 * s;
            src[s] = nullptr; stride[s] = 0; dst[s] = -1;
            if (e < du) { src[s] = qp + 4 * e; stride[s] = p.q_stride; dst[s] = 4 * e; }
            else if (e < 2 * du) { src[s] = kp + 4 * (e - du); stride[s] = p.k_stride; dst[s] = SH::DP + 4 * (e - du); }
            else if (CH && e < 3 * du) { src[s] = wp + 4 * (e - 2 * du); stride[s] = p.w_stride; dst[s] = 2 * SH::DP + 4 * (e - 2 * du); }
            else if (e < rows + vu) { src[s] = vp + 4 * (e - rows); stride[s] = p.v_stride; dst[s] = V + 4 * (e - rows); }
            else if (SH::SCALARS && e == rows + vu) { src[s] = sp; stride[s] = 4 * p.heads; dst[s] = SH::TOKEN - 4; }
            if (dst[s] >= 0) src[s] += t0 * stride[s];
        }
    }
    // the next n tokens into `stage`
    __device__ __forceinline__ void bring(float* stage, int n) {
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            if (dst[s] < 0) continue;
            float* d = stage + dst[s];
            if (n == TB) {
#pragma unroll
                for (int tt = 0; tt < TB; ++tt) { copy16(d + tt * SH::TOKEN, src[s]); src[s] += stride[s]; }
            } else {
                for (int tt = 0; tt < n; ++tt) { copy16(d + tt * SH::TOKEN, src[s]); src[s] += stride[s]; }
            }
        }
    }
};
// The same element by element, for rows of other lengths.
template <typename SH>
__device__ __forceinline__ void bring_elements(const ScanParams& p, const float* qp, const float* kp, const float* wp, const float* vp,
                                               const float* sp, int n_cols, long long tb, int n, float* stage, int lane) {
    constexpr bool CH = SH::ROWS == 3;
    constexpr int V = SH::ROWS * SH::DP;
    const int dim = p.dim;
#pragma unroll 1
    for (int tt = 0; tt < n; ++tt) {
        float* d = stage + tt * SH::TOKEN;
        const long long t = tb + tt;
        for (int e = lane; e < dim; e += 32) {
            copy4(d + e, qp + t * p.q_stride + e);
            copy4(d + SH::DP + e, kp + t * p.k_stride + e);
            if constexpr (CH) copy4(d + 2 * SH::DP + e, wp + t * p.w_stride + e);
        }
        for (int e = lane; e < n_cols; e += 32) copy4(d + V + e, vp + t * p.v_stride + e);
        if (SH::SCALARS && lane < 2) copy4(d + SH::TOKEN - 4 + lane, sp + t * (4 * p.heads) + lane);
    }
}

// grid (ceil(vdim / (WC * warps)), heads, segments), block 32 * (warps + 1)
template <int LR, int RPV, int CC, int TB, int WALK>
__global__ void __launch_bounds__(32 * (MAX_WARPS + 1)) scan_kernel(const ScanParams p, const int wide, const Leftovers left) {
    using SH = WalkShape<LR, RPV, CC, TB, WALK>;
    constexpr bool CH = SH::CH;
    constexpr int DP = SH::DP, WC = SH::WC, NP = RPV * 2, TOKEN = SH::TOKEN, V = SH::ROWS * DP;
    extern __shared__ __align__(16) float ring[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x >> 5) - 1;
    const int seg = blockIdx.z, head = blockIdx.y;
    const int dim = p.dim, vdim = p.vdim, dim4 = (dim + 3) & ~3;
    const int BC = WC * warps, c0 = blockIdx.x * BC;
    // rows beyond dim stay zero in every stage (a decay there multiplies zeros)
    if (DP > dim) {
        const int gap = DP - dim;
        for (int e = threadIdx.x; e < RING * TB * SH::ROWS * gap; e += blockDim.x) {
            const int t = e / (SH::ROWS * gap), i = e % (SH::ROWS * gap);
            ring[t * TOKEN + (i / gap) * DP + dim + i % gap] = 0.f;
        }
    }
    pdl_wait();
    const int t0 = p.cu_seqlens[seg], t1 = p.cu_seqlens[seg + 1];
    if (t0 >= t1) return;
    const int what = left_over(left, p.cu_seqlens, seg, head, p.heads, c0, BC);
    if (what == NOTHING) return;
    const int slot = p.slots[seg];
    if (seg > 0 && slot == p.slots[0]) {                  // a captured step's padding row (a copy of the first row): the state
        for (int e = threadIdx.x; e < (t1 - t0) * BC; e += blockDim.x)      // moves on once; the copy's results are never read
            if (c0 + e % BC < vdim) p.out[(size_t)(t0 + e / BC) * p.out_stride + (size_t)head * vdim + c0 + e % BC] = 0.f;
        return;
    }
    const int n_cols = min(BC, vdim - c0);
    const int n_batches = (t1 - t0 + TB - 1) / TB;

    if (warp == warps) {                                  // the warp that brings the inputs
        const int kvh = head / (p.heads / p.kv_heads);
        const float* qp = p.q + (size_t)kvh * dim;
        const float* kp = p.k + (size_t)kvh * dim;
        const float* vp = p.v + (size_t)head * vdim + c0;
        const float* wp = CH ? p.w + (size_t)head * dim : nullptr;
        const float* sp = SH::SCALARS ? p.scalars + 4 * head : nullptr;
        const auto pump = [&](auto&& bring) {             // bring(batch): starts its copies
#pragma unroll 1
            for (int b = 0; b < RING - 1; ++b) { bring(b); copy_commit(); }
#pragma unroll 1
            for (int b = 0; b < n_batches; ++b) {
                copy_wait<RING - 2>();
                block_barrier(blockDim.x);                // batch b has landed, and every warp is done with batch b - 1
                bring(b + RING - 1);                      // (into the stage that batch b - 1 had)
                copy_commit();
            }
            copy_wait<0>();
        };
        if (wide) {
            Bringer<SH, TB> br(p, qp, kp, wp, vp, sp, n_cols, t0, lane);
            pump([&](int b) { if (b < n_batches) br.bring(ring + (b % RING) * TB * TOKEN, min(TB, t1 - t0 - b * TB)); });
        } else {
            pump([&](int b) {
                if (b < n_batches)
                    bring_elements<SH>(p, qp, kp, wp, vp, sp, n_cols, t0 + (long long)b * TB, min(TB, t1 - t0 - b * TB),
                                       ring + (b % RING) * TB * TOKEN, lane);
            });
        }
        return;
    }

    // the state: value column j = c0 + warp * WC + cl * CC + c, key rows 4 (r + LR i) .. + 3
    const int r = lane % LR, cl = lane / LR;
    float* st = p.state + (size_t)slot * p.slot_stride + (size_t)head * vdim * dim4;
    const int j0 = warp * WC + cl * CC;                   // within the block's columns
    const bool mine = j0 < n_cols && left_column(left, what, seg, head, p.heads, c0 + j0);     // (a lane's columns are in one group of 16)
    f2 S[NP][CC];
#pragma unroll
    for (int c = 0; c < CC; ++c)
#pragma unroll
        for (int i = 0; i < RPV; ++i) {
            const int row = 4 * (r + LR * i);
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < dim4 && j0 + c < n_cols) f = *(const float4*)(st + (size_t)(c0 + j0 + c) * dim4 + row);
            S[2 * i][c] = pack2(f.x, f.y); S[2 * i + 1][c] = pack2(f.z, f.w);
        }

    const float skip = p.skip ? p.skip[head] : 0.f;
    auto token = [&](const float* in, float* o) {         // in: the token's stage
        f2 q[NP], k[NP], w[CH ? NP : 1];
#pragma unroll
        for (int i = 0; i < RPV; ++i) {
            const int row = 4 * (r + LR * i);
            const ulonglong2 a = *(const ulonglong2*)(in + row), b = *(const ulonglong2*)(in + DP + row);
            q[2 * i] = a.x; q[2 * i + 1] = a.y; k[2 * i] = b.x; k[2 * i + 1] = b.y;
            if constexpr (CH) {
                const ulonglong2 d = *(const ulonglong2*)(in + 2 * DP + row);
                w[2 * i] = d.x; w[2 * i + 1] = d.y;
            }
        }
        f2 decay = 0;
        float v[CC];
        if constexpr (CC == 4) { const float4 f = *(const float4*)(in + V + j0); v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; }
        else { const float2 f = *(const float2*)(in + V + j0); v[0] = f.x; v[1] = f.y; }
        if constexpr (!CH) {
            const float2 s = *(const float2*)(in + TOKEN - 4);
            decay = pack2(s.x, s.x);
#pragma unroll
            for (int c = 0; c < CC; ++c) v[c] *= s.y;
        }
#pragma unroll
        for (int c = 0; c < CC; ++c) {
            const f2 v2 = pack2(v[c], v[c]);
            f2 acc = 0;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if constexpr (WALK == PER_CHANNEL_BONUS) {
                    acc = fma2(q[i], S[i][c], acc);
                    S[i][c] = fma2(w[i], S[i][c], mul2(k[i], v2));
                } else if constexpr (WALK == PER_CHANNEL) {
                    S[i][c] = fma2(w[i], S[i][c], mul2(k[i], v2));
                    acc = fma2(q[i], S[i][c], acc);
                } else {
                    S[i][c] = fma2(k[i], v2, mul2(decay, S[i][c]));
                    acc = fma2(q[i], S[i][c], acc);
                }
            }
            float lo, hi;
            unpack2(acc, lo, hi);
            o[c] = lo + hi;
        }
    };

    float* out = p.out + (size_t)t0 * p.out_stride + (size_t)head * vdim + c0 + j0;
    int stage = 0;
#pragma unroll 1
    for (int rest = t1 - t0; rest > 0; rest -= TB) {
        block_barrier(blockDim.x);
        const float* in = ring + stage * (TB * TOKEN);
        stage = stage + 1 == RING ? 0 : stage + 1;
        float o[TB * CC];
        if (rest >= TB) {
#pragma unroll
            for (int tt = 0; tt < TB; ++tt) token(in + tt * TOKEN, o + tt * CC);
        } else {
#pragma unroll
            for (int tt = 0; tt < TB; ++tt) {
                if (tt < rest) token(in + tt * TOKEN, o + tt * CC);
                else
#pragma unroll
                    for (int c = 0; c < CC; ++c) o[tt * CC + c] = 0.f;
            }
        }
        // sums over the LR lanes of the keys; lane r keeps the numbers r * KEEP .. (number n: token n / CC, column n % CC)
#pragma unroll
        for (int h = LR / 2; h >= 1; h >>= 1) {
            const bool up = (r & h) != 0;
#pragma unroll
            for (int i = 0; i < h * SH::KEEP; ++i) {
                const float give = up ? o[i] : o[i + h * SH::KEEP], keep = up ? o[i + h * SH::KEEP] : o[i];
                o[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
            }
        }
#pragma unroll
        for (int i = 0; i < SH::KEEP; ++i) {
            const int num = r * SH::KEEP + i, tt = num / CC, c = num % CC;
            if (tt < rest && mine && j0 + c < n_cols) {
                const float* tok = in + tt * TOKEN;
                out[(long long)tt * p.out_stride + c] =
                    WALK == PER_CHANNEL ? p.out_scale * o[i] : fmaf(CH ? tok[TOKEN - 4] : skip, tok[V + j0 + c], o[i]);
            }
        }
        out += TB * p.out_stride;
    }
#pragma unroll
    for (int c = 0; c < CC; ++c)
#pragma unroll
        for (int i = 0; i < RPV; ++i) {
            const int row = 4 * (r + LR * i);
            if (row < dim4 && mine && j0 + c < n_cols) {
                float4 f;
                unpack2(S[2 * i][c], f.x, f.y); unpack2(S[2 * i + 1][c], f.z, f.w);
                *(float4*)(st + (size_t)(c0 + j0 + c) * dim4 + row) = f;
            }
        }
    pdl_launch_dependents();                              // (late: the next kernel's blocks would only sit and wait)
}

// ---- what a token brings besides q, k and v
// state space: scalars[t, h] = (exp(-exp(A_log[h]) dt), dt, -, -), dt = softplus(a[t, h] + dt_bias[h])
__global__ void __launch_bounds__(128) state_space_gates_kernel(const float* __restrict__ a, long long stride,
                                                                const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                                                float* __restrict__ scalars, long long n, int heads) {
    pdl_wait();
    pdl_launch_dependents();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long t = i / heads;
    const int h = (int)(i % heads);
    const float z = a[t * stride + h] + dt_bias[h];
    const float dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
    *(float4*)(scalars + 4 * i) = make_float4(expf(-expf(a_log[h]) * dt), dt, 0.f, 0.f);
}

// decaying memory: w[t, h, i] = exp(-exp(z + w0)) in place, scalars[t, h, 0] = sum_i q_i u_i k_i.  One warp per (token, head).
__global__ void __launch_bounds__(128) memory_gates_kernel(float* __restrict__ w, long long w_stride, const float* __restrict__ w0,
                                                           const float* __restrict__ q, long long q_stride,
                                                           const float* __restrict__ k, long long k_stride,
                                                           const float* __restrict__ u, float* __restrict__ scalars, long long rows,
                                                           int heads, int dim) {
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const long long t = row / heads;
    const int h = (int)(row % heads);
    float* wr = w + t * w_stride + (size_t)h * dim;
    const float* qr = q + t * q_stride + (size_t)h * dim;
    const float* kr = k + t * k_stride + (size_t)h * dim;
    float s = 0.f;
    for (int i = lane; i < dim; i += 32) {
        wr[i] = expf(-expf(wr[i] + w0[h * dim + i]));
        s = fmaf(qr[i] * u[h * dim + i], kr[i], s);
    }
    s = warp_sum(s);
    if (lane == 0) *(float4*)(scalars + 4 * row) = make_float4(s, 0.f, 0.f, 0.f);
}

// gated linear attention: w[t, c] = sigmoid(z)^(1/tau) with z = sum_r a[t, r] A_2[r, c] + b[c] for the channels c of all heads.
// A thread has one channel of DECAY_TOKENS tokens (8 in prompts, 1 in steps of few tokens); the sum runs over r in ascending order.
constexpr int DECAY_RANK = 64;                            // (the short vectors of a block's tokens pass through in pieces)
template <int DECAY_TOKENS>
__global__ void __launch_bounds__(128) channel_decays_kernel(const float* __restrict__ a, long long a_stride, const float* __restrict__ a2,
                                                             const float* __restrict__ b, float* __restrict__ w, long long w_stride,
                                                             int n_tokens, int n, int rank, float inv_tau) {
    __shared__ float a_s[DECAY_TOKENS][DECAY_RANK];
    pdl_wait();
    pdl_launch_dependents();
    const int c = blockIdx.x * 128 + threadIdx.x, t0 = blockIdx.y * DECAY_TOKENS, nt = min(DECAY_TOKENS, n_tokens - t0);
    float z[DECAY_TOKENS];
#pragma unroll
    for (int t = 0; t < DECAY_TOKENS; ++t) z[t] = 0.f;
    for (int r0 = 0; r0 < rank; r0 += DECAY_RANK) {
        const int nr = min(DECAY_RANK, rank - r0);
        if (r0 > 0) __syncthreads();
        for (int e = threadIdx.x; e < DECAY_TOKENS * nr; e += 128) {
            const int t = e / nr, r = e % nr;
            a_s[t][r] = t < nt ? a[(long long)(t0 + t) * a_stride + r0 + r] : 0.f;
        }
        __syncthreads();
        if (c < n) {
#pragma unroll 16
            for (int r = 0; r < nr; ++r) {
                const float v = a2[(size_t)(r0 + r) * n + c];
#pragma unroll
                for (int t = 0; t < DECAY_TOKENS; ++t) z[t] = fmaf(a_s[t][r], v, z[t]);
            }
        }
    }
    if (c >= n) return;
    const float bias = b[c];
#pragma unroll
    for (int t = 0; t < DECAY_TOKENS; ++t) {
        if (t >= nt) break;
        const float y = z[t] + bias;                      // log sigmoid(y) = -(max(-y, 0) + log(1 + e^-|y|))
        w[(long long)(t0 + t) * w_stride + c] = expf(-inv_tau * (fmaxf(-y, 0.f) + log1pf(expf(-fabsf(y)))));
    }
}

template <int LR, int RPV, int CC, int TB, int WALK>
int launch_scan(const ScanParams& p, int wide, const Leftovers& left, cudaStream_t st) {
    using SH = WalkShape<LR, RPV, CC, TB, WALK>;
    // four walking warps a block, fewer where a step has so few (segment, head) pairs that more and smaller blocks spread better
    int warps = MAX_WARPS;
    while (warps > 1 && ((long long)((p.vdim + SH::WC * warps - 1) / (SH::WC * warps)) * p.heads * p.n_segments < 148 ||
                         SH::WC * (warps / 2) >= p.vdim)) warps /= 2;
    const size_t bytes = (size_t)RING * TB * SH::TOKEN * sizeof(float);
    auto kernel = scan_kernel<LR, RPV, CC, TB, WALK>;
    if (bytes > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
        return SPITE_LAUNCH_FAILED;
    dim3 grid((p.vdim + SH::WC * warps - 1) / (SH::WC * warps), p.heads, p.n_segments);
    // A step of single tokens is launched as a programmatic dependent; a longer walk in the ordinary way: started early, its
    // blocks would take the multiprocessors that the kernel before frees first, several to one, for the whole walk.
    if (p.n_tokens == p.n_segments) SPITE_LAUNCH(kernel, grid, 32 * (warps + 1), bytes, st, p, wide, left);
    else kernel<<<grid, 32 * (warps + 1), bytes, st>>>(p, wide, left);
    return spite_launch_status();
}

template <int WALK>
int choose_scan(const ScanParams& p, cudaStream_t st, const Leftovers& left = {}) {
    constexpr bool CH = WALK != PER_HEAD;
    const auto al = [](const void* x) { return ((uintptr_t)x & 15) == 0; };
    const int wide = p.dim % 4 == 0 && p.vdim % 4 == 0 && p.q_stride % 4 == 0 && p.k_stride % 4 == 0 && p.v_stride % 4 == 0 &&
                     al(p.q) && al(p.k) && al(p.v) && (WALK == PER_CHANNEL || al(p.scalars)) && (!CH || (p.w_stride % 4 == 0 && al(p.w)));
    if (p.dim <= 32) return launch_scan<8, 1, 2, 8, WALK>(p, wide, left, st);
    if (p.dim <= 64) return launch_scan<8, 2, 2, 8, WALK>(p, wide, left, st);
    if (p.dim <= 128) return launch_scan<8, 4, 2, 8, WALK>(p, wide, left, st);
    if (p.dim <= 256) return launch_scan<16, 4, 2, 8, WALK>(p, wide, left, st);
    return launch_scan<32, 4, 4, 8, WALK>(p, wide, left, st);
}

// ---- what the walk in chunks needs that does not depend on the state
// q and k of a chunk (a warp has the tokens warp, warp + 8, ..., a lane the elements lane, lane + 32, ...; 256 threads) into split tiles;
// q_t . k_s into `scores`, the sizes of the tokens' rows into `q_size`, `k_size`.  Returns whether a number is not finite (of the warp's).
template <int DP>
__device__ __forceinline__ bool split_tiles(const float* q, long long q_stride, const float* k, long long k_stride, int len, int dim, __half* tiles,
                                            float (*scores)[36], float* q_size, float* k_size) {
    constexpr int E = DP / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    float qv[4][E], kv[4][E];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int t = warp + 8 * i, d = lane + 32 * e;
            const bool on = t < len && d < dim;
            qv[i][e] = on ? q[t * q_stride + d] : 0.f;
            kv[i][e] = on ? k[t * k_stride + d] : 0.f;
        }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        unsigned lq = 0, lk = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) { lq = max(lq, abs_bits(qv[i][e])); lk = max(lk, abs_bits(kv[i][e])); }
        lq = __reduce_max_sync(0xffffffffu, lq);
        lk = __reduce_max_sync(0xffffffffu, lk);
        bad |= max(lq, lk) >= 0x7f800000u;
        const Scale sq = scale_of(lq), sk = scale_of(lk);
        if (lane == 0) { q_size[warp + 8 * i] = sq.size; k_size[warp + 8 * i] = sk.size; }
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int at = tile_at<DP>(warp + 8 * i, lane + 32 * e);
            split1(qv[i][e] * sq.up, tiles[at], tiles[CT * DP + at]);
            split1(kv[i][e] * sk.up, tiles[2 * CT * DP + at], tiles[3 * CT * DP + at]);
        }
    }
    __syncthreads();
    const int m = warp & 1, n = warp >> 1;                // sixteen tokens t and eight tokens s a warp
    float main[4] = {}, cross[4] = {};
    if (n < 2 || m == 1) {
#pragma unroll 4
        for (int k16 = 0; k16 < DP / 16; k16 += 2) {
            unsigned bh[4], bl[4], ah[4], al[4];
            ldsm(bh, tiles + 2 * CT * DP + tile_at<DP>(8 * n + (lane & 7), 16 * k16 + 8 * (lane >> 3)));
            ldsm(bl, tiles + 3 * CT * DP + tile_at<DP>(8 * n + (lane & 7), 16 * k16 + 8 * (lane >> 3)));
            ldsm_left<DP>(ah, tiles, 16 * m, 16 * k16, lane);
            ldsm_left<DP>(al, tiles + CT * DP, 16 * m, 16 * k16, lane);
            mma3(main, cross, ah, al, bh[0], bh[1], bl[0], bl[1]);
            ldsm_left<DP>(ah, tiles, 16 * m, 16 * k16 + 16, lane);
            ldsm_left<DP>(al, tiles + CT * DP, 16 * m, 16 * k16 + 16, lane);
            mma3(main, cross, ah, al, bh[2], bh[3], bl[2], bl[3]);
        }
    }
    const float2 ks = *(const float2*)(k_size + 8 * n + 2 * t4);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float qs = q_size[16 * m + g + 8 * r];
        *(float2*)&scores[16 * m + g + 8 * r][8 * n + 2 * t4] = make_float2(sum2(main[2 * r], cross[2 * r]) * qs * ks.x,
                                                                             sum2(main[2 * r + 1], cross[2 * r + 1]) * qs * ks.y);
    }
    return bad;
}
template <int DP> __device__ __forceinline__ void store_tiles(__half* to, const __half* tiles) {
    uint4* dst = reinterpret_cast<uint4*>(to);
    const uint4* src = reinterpret_cast<const uint4*>(tiles);
#pragma unroll 4
    for (int e = threadIdx.x; e < 4 * CT * DP / 8; e += blockDim.x) dst[e] = src[e];
}

// One decay a head.  A block has a chunk of one q/k head and up to SSM_HEADS of the heads that share it, a warp one of them at a time.
constexpr int SSM_HEADS = 16;
template <int DP> struct StateSpaceChunkSmem {
    __half tiles[4 * CT * DP];
    float scores[CT][36];
    double b[8][CT];
    float dt[8][CT], q_size[CT], k_size[CT];
};
template <int DP>
__global__ void __launch_bounds__(256) state_space_chunk_kernel(const ScanParams p, const float* __restrict__ a, long long a_stride,
                                                                const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                                                float* __restrict__ scalars, const Made out, int slices) {
    using Rec = Record<HEAD_DECAY, DP>;
    extern __shared__ __align__(16) unsigned char smem_bytes[];
    auto& sm = *reinterpret_cast<StateSpaceChunkSmem<DP>*>(smem_bytes);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = p.heads / p.kv_heads, kvh = blockIdx.y / slices, slice = blockIdx.y % slices;
    const int h0 = kvh * group + slice * SSM_HEADS, h1 = min(h0 + SSM_HEADS, (kvh + 1) * group);
    pdl_wait();
    pdl_launch_dependents();
    Place pl;
    if (!find_chunk<ALL>(out.numbering, p.cu_seqlens, p.n_segments, blockIdx.x, pl)) return;
    const int first = pl.first, len = min(CT, pl.end - first);
    const bool brief = pl.at < 0;                         // walked token by token: the tokens' scalars alone
    if (!brief && first == pl.begin)
        for (int h = h0 + warp; h < h1; h += 8) clear_marks(out.columns, out.column_groups, pl.seg, h, p.heads, lane, 32);
    bool bad = false;
    if (!brief) {
        bad = split_tiles<DP>(p.q + (size_t)first * p.q_stride + (size_t)kvh * p.dim, p.q_stride, p.k + (size_t)first * p.k_stride + (size_t)kvh * p.dim,
                              p.k_stride, len, p.dim, sm.tiles, sm.scores, sm.q_size, sm.k_size);
        if (slice == 0) store_tiles<DP>(out.qk + ((size_t)pl.at * p.kv_heads + kvh) * (4 * CT * DP), sm.tiles);
        bad = __syncthreads_or(bad);
    }
    for (int h = h0 + warp; h < h1; h += 8) {             // a lane a token
        float dt = 0.f, log_decay = 0.f;
        bool lost = false;
        if (lane < len) {
            const float z = a[(long long)(first + lane) * a_stride + h] + dt_bias[h];
            dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
            log_decay = -expf(a_log[h]) * dt;
            lost = !(dt < 3e38f) || !(log_decay <= 0.f);
            *(float4*)(scalars + 4 * ((size_t)(first + lane) * p.heads + h)) = make_float4(expf(log_decay), dt, 0.f, 0.f);
        }
        if (brief) continue;
        const double b = prefix_sum((double)bounded_log(log_decay), lane), last = __shfl_sync(0xffffffffu, b, len - 1);
        __syncwarp();
        sm.b[warp][lane] = b;
        sm.dt[warp][lane] = dt;
        __syncwarp();
        float x[CT];                                      // a lane has a row of scores
        unsigned largest = 0;
#pragma unroll
        for (int s = 0; s < CT; s += 4) {
            const float4 gs = *(const float4*)&sm.scores[lane][s];
            const float row[4] = {gs.x, gs.y, gs.z, gs.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[s + i] = s + i <= lane ? row[i] * expf((float)(b - sm.b[warp][s + i])) * sm.dt[warp][s + i] : 0.f;
                largest = max(largest, abs_bits(x[s + i]));
            }
        }
        const Scale sp = scale_of(largest);
        const size_t at_head = (size_t)pl.at * p.heads + h;
        __half* scores = out.scores + at_head * (2 * CT * CT);
#pragma unroll
        for (int s = 0; s < CT; s += 8) {
            uint4 hi, lo;
            split2(x[s] * sp.up, x[s + 1] * sp.up, hi.x, lo.x);
            split2(x[s + 2] * sp.up, x[s + 3] * sp.up, hi.y, lo.y);
            split2(x[s + 4] * sp.up, x[s + 5] * sp.up, hi.z, lo.z);
            split2(x[s + 6] * sp.up, x[s + 7] * sp.up, hi.w, lo.w);
            *(uint4*)(scores + score_at(lane, s)) = hi;
            *(uint4*)(scores + CT * CT + score_at(lane, s)) = lo;
        }
        lost = __any_sync(0xffffffffu, lost || bad || largest >= 0x7f800000u);
        float* rec = out.records + at_head * Rec::FLOATS;
        rec[Rec::G + lane] = expf((float)b);
        rec[Rec::W + lane] = dt * expf((float)(last - b)) * sm.k_size[lane];          // (beyond the chunk's tokens dt is zero)
        rec[Rec::Q_SIZE + lane] = sm.q_size[lane];
        rec[Rec::P_SIZE + lane] = sp.size;
        if (lane < 8) rec[Rec::SCALARS + lane] = lane == DECAY ? expf((float)last) : lane == BAD && lost ? 1.f : 0.f;
    }
}

// A decay per key channel: one block a (chunk, head), 256 threads.  Scores of two tokens in the same half of the chunk are summed with
// the products of the decays between them; those of the later half with the earlier are one product of operands that are brought to
// the decays at the border.  BONUS (the decaying memory): a token's read-out sees the state before its own write, plus the bonus.
template <int DP> struct KeyDecayChunkSmem {
    __half tiles[4 * CT * DP], off[2 * CT * DP];          // `off`: rows 0 .. 15 k of the first half, 16 .. 31 q of the second, brought to the border
    float q[CT][DP + 4], k[CT][DP + 4], w[CT][DP + 4];
    float P[CT][36];
    float part[256 / DP][DP];                             // sums of log decays of a thread's tokens
    unsigned largest[3][CT];                              // of the rows of q and of k in `tiles`, of those of `off`
    int bad;
};
template <int DP, bool BONUS>
__global__ void __launch_bounds__(256) key_decay_chunk_kernel(const ScanParams p, const Made out) {
    using Rec = Record<KEY_DECAY, DP>;
    constexpr int PARTS = 256 / DP, TN = CT / PARTS;      // a thread has a channel of TN tokens
    extern __shared__ __align__(16) unsigned char smem_bytes[];
    auto& sm = *reinterpret_cast<KeyDecayChunkSmem<DP>*>(smem_bytes);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, head = blockIdx.y, dim = p.dim;
    pdl_wait();
    pdl_launch_dependents();
    Place pl;
    if (!find_chunk<NUMBERED>(out.numbering, p.cu_seqlens, p.n_segments, blockIdx.x, pl) || pl.at < 0) return;
    const int first = pl.first, len = min(CT, pl.end - first);
    if (first == pl.begin) clear_marks(out.columns, out.column_groups, pl.seg, head, p.heads, tid, 256);
    if (tid < 3 * CT) sm.largest[tid / CT][tid % CT] = 0;
    if (tid == 0) sm.bad = 0;
    const size_t at_head = (size_t)pl.at * p.heads + head;
    const int ch = tid % DP, part = tid / DP;
    float qv[TN], kv[TN], lw[TN];                         // q, k and the log decays
    bool bad = false;
    {
        const float* q = p.q + (size_t)first * p.q_stride + (size_t)head * dim + ch;
        const float* k = p.k + (size_t)first * p.k_stride + (size_t)head * dim + ch;
        const float* w = p.w + (size_t)first * p.w_stride + (size_t)head * dim + ch;
        float wv[TN];
#pragma unroll
        for (int i = 0; i < TN; ++i) {
            const int t = part * TN + i;
            const bool on = t < len && ch < dim;
            qv[i] = on ? q[(size_t)t * p.q_stride] : 0.f;
            kv[i] = on ? k[(size_t)t * p.k_stride] : 0.f;
            wv[i] = on ? w[(size_t)t * p.w_stride] : 1.f;
        }
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < TN; ++i) {
            const int t = part * TN + i;
            sm.q[t][ch] = qv[i]; sm.k[t][ch] = kv[i]; sm.w[t][ch] = wv[i];
            bad |= !(wv[i] >= 0.f && wv[i] <= 1.f);
            lw[i] = bounded_log(logf(wv[i]));
            sum += lw[i];
        }
        sm.part[part][ch] = sum;
    }
    for (int e = tid; e < CT * CT; e += 256) sm.P[e / CT][e % CT] = 0.f;
    __syncthreads();
    {
        // Sums of log decays from the chunk's start to a token, from behind it to the end, and between it and the border: each is made
        // from its own end, so that a small one has no large one's rounding in it.
        constexpr int HALF = PARTS / 2;
        float before = 0.f, after = 0.f, inner = 0.f, last = 0.f;     // over the parts before, behind, and between this one and the border
#pragma unroll
        for (int i = 0; i < PARTS; ++i) {
            const float s = sm.part[i][ch];
            if (i < part) before += s;
            if (i > part) after += s;
            if (part < HALF ? i > part && i < HALF : i >= HALF && i < part) inner += s;
            last += s;
        }
        float qs[TN], ks[TN], os[TN];
        float run = 0.f, back = 0.f;
#pragma unroll
        for (int i = 0; i < TN; ++i) {                    // (a token of the memory is read before its own decay)
            if (!BONUS) run += lw[i];
            qs[i] = qv[i] * expf(before + run);
            if (part >= HALF) os[i] = qv[i] * expf(inner + run);
            if (BONUS) run += lw[i];
        }
#pragma unroll
        for (int i = TN - 1; i >= 0; --i) {
            ks[i] = kv[i] * expf(after + back);
            if (part < HALF) os[i] = kv[i] * expf(inner + back);
            back += lw[i];
        }
#pragma unroll
        for (int i = 0; i < TN; ++i) {
            const unsigned lq = __reduce_max_sync(0xffffffffu, abs_bits(qs[i])), lk = __reduce_max_sync(0xffffffffu, abs_bits(ks[i])),
                           lo = __reduce_max_sync(0xffffffffu, abs_bits(os[i]));
            bad |= max(abs_bits(qv[i]), abs_bits(kv[i])) >= 0x7f800000u;
            if (lane < 3) atomicMax(&sm.largest[lane][part * TN + i], lane == 0 ? lq : lane == 1 ? lk : lo);
        }
        if (bad) sm.bad = 1;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TN; ++i) {
            const int t = part * TN + i, at = tile_at<DP>(t, ch);
            split1(qs[i] * scale_of(sm.largest[0][t]).up, sm.tiles[at], sm.tiles[CT * DP + at]);
            split1(ks[i] * scale_of(sm.largest[1][t]).up, sm.tiles[2 * CT * DP + at], sm.tiles[3 * CT * DP + at]);
            split1(os[i] * scale_of(sm.largest[2][t]).up, sm.off[at], sm.off[CT * DP + at]);
        }
        float* rec = out.records + at_head * Rec::FLOATS;
        if (part == 0) rec[Rec::KEYS + ch] = ch < dim ? expf(last) : 0.f;
        if (tid < CT) { rec[Rec::Q_SIZE + tid] = scale_of(sm.largest[0][tid]).size; rec[Rec::W + tid] = scale_of(sm.largest[1][tid]).size; }
    }
    // ---- scores within a half of the chunk: a warp has four tokens s, its lanes the channels (four tokens in a row, with what
    // a token t brings read once: 58 against 48 us for 2,048 tokens of 32 heads of 64, for its 64 sums a lane)
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const int s = warp + 8 * i, end = (s & 16) + 16;
        constexpr int C2 = DP / 64;                       // pairs of channels a lane
        float2 kf[C2];
        float o[16];
#pragma unroll
        for (int c = 0; c < C2; ++c) kf[c] = *(const float2*)&sm.k[s][2 * lane + 64 * c];
#pragma unroll
        for (int j = 0; j < 16; ++j) {                    // token s + j
            o[j] = 0.f;
            if (s + j < end) {
#pragma unroll
                for (int c = 0; c < C2; ++c) {
                    const float2 w = *(const float2*)&sm.w[s + j][2 * lane + 64 * c], q = *(const float2*)&sm.q[s + j][2 * lane + 64 * c];
                    if (!BONUS && j) { kf[c].x *= w.x; kf[c].y *= w.y; }
                    if (!BONUS || j) { o[j] = fmaf(q.x, kf[c].x, o[j]); o[j] = fmaf(q.y, kf[c].y, o[j]); }
                    if (BONUS && j) { kf[c].x *= w.x; kf[c].y *= w.y; }
                }
            }
        }
#pragma unroll
        for (int h = 8; h >= 1; h >>= 1) {
            const bool up = (lane & h) != 0;
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const float give = up ? o[j] : o[j + h], keep = up ? o[j + h] : o[j];
                o[j] = keep + __shfl_xor_sync(0xffffffffu, give, h);
            }
        }
        float x = o[0] + __shfl_xor_sync(0xffffffffu, o[0], 16);
        const int t = s + lane;
        if (lane < 16 && t < end) {
            if (BONUS && lane == 0) x = t < len ? p.scalars[4 * ((size_t)(first + t) * p.heads + head)] : 0.f;
            sm.P[t][s] = x;
        }
    }
    __syncthreads();
    // ---- scores of the second half with the first: two warps, eight tokens s each
    if (warp < 2) {
        const int s = 8 * warp + 2 * (lane & 3);
        const float s0 = scale_of(sm.largest[2][s]).size, s1 = scale_of(sm.largest[2][s + 1]).size;
        float main[4] = {}, cross[4] = {};
#pragma unroll
        for (int k = 0; k < DP / 16; k += 2) {
            unsigned bh[4], bl[4], ah[4], al[4];
            ldsm(bh, sm.off + tile_at<DP>(8 * warp + (lane & 7), 16 * k + 8 * (lane >> 3)));
            ldsm(bl, sm.off + CT * DP + tile_at<DP>(8 * warp + (lane & 7), 16 * k + 8 * (lane >> 3)));
            ldsm_left<DP>(ah, sm.off, 16, 16 * k, lane);
            ldsm_left<DP>(al, sm.off + CT * DP, 16, 16 * k, lane);
            mma3(main, cross, ah, al, bh[0], bh[1], bl[0], bl[1]);
            ldsm_left<DP>(ah, sm.off, 16, 16 * k + 16, lane);
            ldsm_left<DP>(al, sm.off + CT * DP, 16, 16 * k + 16, lane);
            mma3(main, cross, ah, al, bh[2], bh[3], bl[2], bl[3]);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = 16 + (lane >> 2) + 8 * r;
            const float st = scale_of(sm.largest[2][t]).size;
            *(float2*)&sm.P[t][s] = make_float2(sum2(main[2 * r], cross[2 * r]) * st * s0, sum2(main[2 * r + 1], cross[2 * r + 1]) * st * s1);
        }
    }
    store_tiles<DP>(out.qk + at_head * (4 * CT * DP), sm.tiles);
    __syncthreads();
    const int t = tid >> 3, s = 4 * (tid & 7);
    const float4 x = *(const float4*)&sm.P[t][s];
    unsigned largest = quad_max(max(max(abs_bits(x.x), abs_bits(x.y)), max(abs_bits(x.z), abs_bits(x.w))));
    largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, 4));
    const Scale sp = scale_of(largest);
    uint2 h, l;
    split2(x.x * sp.up, x.y * sp.up, h.x, l.x);
    split2(x.z * sp.up, x.w * sp.up, h.y, l.y);
    __half* scores = out.scores + at_head * (2 * CT * CT) + score_at(t, s);
    *(uint2*)scores = h;
    *(uint2*)(scores + CT * CT) = l;
    float* rec = out.records + at_head * Rec::FLOATS;
    if ((tid & 7) == 0) rec[Rec::P_SIZE + t] = sp.size;
    const bool lost = __syncthreads_or(largest >= 0x7f800000u);
    if (tid < 8) rec[Rec::SCALARS + tid] = tid == BAD && (sm.bad || lost) ? 1.f : 0.f;
}

inline Layout scan_layout(bool per_channel, int dim, int vdim, int heads, int kv_heads, int n_chunks, int n_segments) {
    const int dp = dim <= 64 ? 64 : 128;
    const int record = !per_channel ? Record<HEAD_DECAY, 64>::FLOATS : dp == 64 ? Record<KEY_DECAY, 64>::FLOATS : Record<KEY_DECAY, 128>::FLOATS;
    return layout_of(dp, record, heads, kv_heads, vdim, n_chunks, n_segments, false, 0);
}
inline chunk::Walk scan_walk(const ScanParams& p, const Made& out) {
    chunk::Walk w = walk_of(out);
    const int dim4 = (p.dim + 3) & ~3;
    w.v = p.v; w.v_stride = p.v_stride;
    w.out = p.out; w.out_stride = p.out_stride;
    w.state = p.state; w.slot_stride = p.slot_stride; w.head_stride = (long long)p.vdim * dim4;
    w.key_stride = 1; w.col_stride = dim4;
    w.cu_seqlens = p.cu_seqlens; w.slots = p.slots;
    w.n_segments = p.n_segments; w.heads = p.heads; w.qk_heads = p.kv_heads; w.dim = p.dim; w.vdim = p.vdim;
    return w;
}
template <int DP>
int launch_state_space_chunks(const ScanParams& p, const float* a, long long a_stride, const float* a_log, const float* dt_bias, const Made& out,
                              cudaStream_t st) {
    auto prep = state_space_chunk_kernel<DP>;
    constexpr int bytes = (int)sizeof(StateSpaceChunkSmem<DP>);
    if (cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return SPITE_LAUNCH_FAILED;
    const int slices = (p.heads / p.kv_heads + SSM_HEADS - 1) / SSM_HEADS;
    // (every chunk of the step, also of segments that go token by token: their tokens' scalars come from here)
    SPITE_LAUNCH(prep, dim3(p.n_tokens / CT + p.n_segments, p.kv_heads * slices), 256, bytes, st, p, a, a_stride, a_log, dt_bias, (float*)p.scalars, out, slices);
    if (cudaGetLastError() != cudaSuccess) return SPITE_LAUNCH_FAILED;
    chunk::Walk w = scan_walk(p, out);
    w.skip = p.skip;
    // 32 columns a block: two blocks of four warps on a multiprocessor (three up to 64 keys) wait for each other's barriers less than one of
    // eight with 64 columns does.  us, 64 / 32 columns, the same bits: 128 heads of 128 x 64, one request of 2,048 tokens 199 / 175, five of 410
    // 224 / 195; 64 heads, five of 410 134 / 117; 64 x 64, 64 heads, three of 666 79 / 61; 16 columns 253 in the first.
    // 64 where all blocks are resident at once that way and not with 32: of blocks for up to 64 keys a multiprocessor holds three with 32
    // columns, two with 64.  With the first kernel, 64 / 32: 64 heads of 64 x 64, four of 2,048 288 / 325, 16 heads of 64 x 128, eight of 2,048
    // 366 / 403, eight of 256 69 / 75; with half or twice the blocks 187 / 177 and 538 / 521, 228 / 218; of 128 x 128, as many blocks 579 / 532.
    if constexpr (DP == 64) {
        const long long groups = (long long)p.heads * out.numbering.segments;
        if ((p.vdim + 63) / 64 * groups <= 2 * 148 && (p.vdim + 31) / 32 * groups > 3 * 148) return launch_walk<DP / 2, 2, 4, HEAD_DECAY>(w, s_waits, st);
    }
    return launch_walk<DP / 2, 2, 2, HEAD_DECAY>(w, s_waits, st);
}
template <int DP, bool BONUS>
int launch_key_decay_chunks(const ScanParams& p, const Made& out, int n_chunks, cudaStream_t st) {
    auto prep = key_decay_chunk_kernel<DP, BONUS>;
    constexpr int bytes = (int)sizeof(KeyDecayChunkSmem<DP>);
    if (cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return SPITE_LAUNCH_FAILED;
    SPITE_LAUNCH(prep, dim3(n_chunks, p.heads), 256, bytes, st, p, out);
    if (cudaGetLastError() != cudaSuccess) return SPITE_LAUNCH_FAILED;
    chunk::Walk w = scan_walk(p, out);
    w.out_scale = BONUS ? 1.f : p.out_scale;
    // (32 columns a block: 32 heads of 64 x 128, five requests of 2,048 tokens together 73 us, four of 2,048 each 258; measured with one
    // scale a tile 62 and 231, with 64 columns 68 and 205)
    return launch_walk<32, DP / 32, 2, KEY_DECAY>(w, s_waits, st);
}
template <bool BONUS, int WALK>
int key_decay_in_chunks(const ScanParams& p, void* scratch, int n_chunks, int min_tokens, cudaStream_t st) {
    const Layout l = scan_layout(true, p.dim, p.vdim, p.heads, p.heads, n_chunks, p.n_segments);
    const Made out = made_at(scratch, l, min_tokens, n_chunks, p.n_segments, p.n_long);
    const int rc = p.dim <= 64 ? launch_key_decay_chunks<64, BONUS>(p, out, n_chunks, st) : launch_key_decay_chunks<128, BONUS>(p, out, n_chunks, st);
    if (rc != SPITE_OK) return rc;
    return choose_scan<WALK>(p, st, leftovers_of(out, l, p.heads, Record<KEY_DECAY, 64>::SCALARS));
}

// the working memory of a call in chunks: refused before anything is launched
int check_chunks(const ScanParams& p, const void* scratch, int n_chunks, int min_tokens) {
    if (!scratch || ((uintptr_t)scratch & 15) || n_chunks < 1 || min_tokens < 1) return SPITE_BAD_ARG;
    return p.dim > 128 ? SPITE_UNSUPPORTED : SPITE_OK;
}

int check_scan(const ScanParams* p) {
    if (!p || !p->q || !p->k || !p->v || !p->out || !p->state || !p->cu_seqlens || !p->slots) return SPITE_BAD_ARG;
    if (p->n_segments < 0 || p->n_tokens < 0 || p->heads < 1 || p->kv_heads < 1 || p->heads % p->kv_heads || p->dim < 1 || p->vdim < 1)
        return SPITE_BAD_ARG;
    const long long dim4 = (p->dim + 3) & ~3;
    if (p->slot_stride < (long long)p->heads * p->vdim * dim4 || p->out_stride < (long long)p->heads * p->vdim) return SPITE_BAD_ARG;
    if (p->q_stride < 1 || p->k_stride < 1 || p->v_stride < 1) return SPITE_BAD_ARG;
    if (p->slot_stride % 4 || ((uintptr_t)p->state & 15)) return SPITE_UNSUPPORTED;      // the state moves in 16-byte groups
    if (p->dim > 512 || p->heads > 65535 || p->n_segments > 65535) return SPITE_UNSUPPORTED;
    return SPITE_OK;
}

}  // namespace

// Bytes of working memory that the three walks in chunks need for a step of `n_chunks` chunks of 32 tokens; -2: sizes they do not take.
SPITE_API long long spite_scan_chunk_bytes(int per_channel, int dim, int vdim, int heads, int kv_heads, int n_chunks, int n_segments) {
    if (dim < 1 || vdim < 1 || heads < 1 || kv_heads < 1 || n_chunks < 0 || n_segments < 0) return SPITE_BAD_ARG;
    if (dim > 128) return SPITE_UNSUPPORTED;
    return scan_layout(per_channel != 0, dim, vdim, heads, kv_heads, n_chunks, n_segments).bytes;
}

// `a` [tokens, heads] with rows of a_stride: the projection's step columns; p->scalars is filled here
static int check_state_space(const ScanParams* p, const float* a, long long a_stride, const float* a_log, const float* dt_bias) {
    const int chk = check_scan(p);
    if (chk != SPITE_OK) return chk;
    return !a || !a_log || !dt_bias || !p->scalars || p->w || a_stride < p->heads ? SPITE_BAD_ARG : SPITE_OK;
}
// Segments of at least `min_tokens` tokens in chunks of 32, the others token by token, and those that the working memory, made for
// `n_chunks` chunks, has no place for (in all three).
SPITE_API int spite_state_space_scan_chunked(const ScanParams* p, const float* a, long long a_stride, const float* a_log, const float* dt_bias,
                                             void* scratch, int n_chunks, int min_tokens, void* stream) {
    int chk = check_state_space(p, a, a_stride, a_log, dt_bias);
    if (chk == SPITE_OK) chk = check_chunks(*p, scratch, n_chunks, min_tokens);
    if (chk != SPITE_OK) return chk;
    if (p->n_segments == 0 || p->n_tokens == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const Layout l = scan_layout(false, p->dim, p->vdim, p->heads, p->kv_heads, n_chunks, p->n_segments);
    const Made out = made_at(scratch, l, min_tokens, n_chunks, p->n_segments, p->n_long);
    const int rc = p->dim <= 64 ? launch_state_space_chunks<64>(*p, a, a_stride, a_log, dt_bias, out, st)
                                : launch_state_space_chunks<128>(*p, a, a_stride, a_log, dt_bias, out, st);
    if (rc != SPITE_OK) return rc;
    return choose_scan<PER_HEAD>(*p, st, leftovers_of(out, l, p->heads, Record<HEAD_DECAY, 64>::SCALARS));
}
SPITE_API int spite_state_space_scan(const ScanParams* p, const float* a, long long a_stride, const float* a_log,
                                     const float* dt_bias, void* stream) {
    const int chk = check_state_space(p, a, a_stride, a_log, dt_bias);
    if (chk != SPITE_OK) return chk;
    if (p->n_segments == 0 || p->n_tokens == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long n = (long long)p->n_tokens * p->heads;
    SPITE_LAUNCH(state_space_gates_kernel, (int)((n + 127) / 128), 128, 0, st, a, a_stride, a_log, dt_bias, (float*)p->scalars, n, p->heads);
    if (cudaGetLastError() != cudaSuccess) return SPITE_LAUNCH_FAILED;
    return choose_scan<PER_HEAD>(*p, st);
}

// p->w holds the decay's pre-activations on entry and the decays afterwards; `u` and `w0` [heads * dim]
static int decay_scan(const ScanParams* p, const float* w0, const float* u, bool chunks, void* scratch, int n_chunks, int min_tokens, void* stream) {
    int chk = check_scan(p);
    if (chk == SPITE_OK && chunks) chk = check_chunks(*p, scratch, n_chunks, min_tokens);
    if (chk != SPITE_OK) return chk;
    if (!w0 || !u || !p->scalars || !p->w || p->w_stride < (long long)p->heads * p->dim || p->kv_heads != p->heads || p->skip) return SPITE_BAD_ARG;
    if (p->n_segments == 0 || p->n_tokens == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long rows = (long long)p->n_tokens * p->heads;
    if ((rows + 3) / 4 > 0x7fffffffLL) return SPITE_UNSUPPORTED;
    SPITE_LAUNCH(memory_gates_kernel, (int)((rows + 3) / 4), 128, 0, st, (float*)p->w, p->w_stride, w0, p->q, p->q_stride, p->k,
                 p->k_stride, u, (float*)p->scalars, rows, p->heads, p->dim);
    if (cudaGetLastError() != cudaSuccess) return SPITE_LAUNCH_FAILED;
    if (chunks) return key_decay_in_chunks<true, PER_CHANNEL_BONUS>(*p, scratch, n_chunks, min_tokens, st);
    return choose_scan<PER_CHANNEL_BONUS>(*p, st);
}
SPITE_API int spite_decay_scan(const ScanParams* p, const float* w0, const float* u, void* stream) {
    return decay_scan(p, w0, u, false, nullptr, 0, 0, stream);
}
SPITE_API int spite_decay_scan_chunked(const ScanParams* p, const float* w0, const float* u, void* scratch, int n_chunks, int min_tokens, void* stream) {
    return decay_scan(p, w0, u, true, scratch, n_chunks, min_tokens, stream);
}

// p->w [tokens, heads * dim] receives the decays, from the short vectors `a` [tokens, rank] (rows of a_stride), `a2` [rank,
// heads * dim] and `b` [heads * dim]
static int gated_linear_scan(const ScanParams* p, const float* a, long long a_stride, const float* a2, const float* b, int rank, float tau,
                             bool chunks, void* scratch, int n_chunks, int min_tokens, void* stream) {
    int chk = check_scan(p);
    if (chk == SPITE_OK && chunks) chk = check_chunks(*p, scratch, n_chunks, min_tokens);
    if (chk != SPITE_OK) return chk;
    if (!a || !a2 || !b || rank < 1 || a_stride < rank || !(tau > 0.f) || !(p->out_scale == p->out_scale)) return SPITE_BAD_ARG;
    if (!p->w || p->w_stride < (long long)p->heads * p->dim || p->kv_heads != p->heads || p->skip) return SPITE_BAD_ARG;
    if (p->n_segments == 0 || p->n_tokens == 0) return SPITE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int n = p->heads * p->dim;
    const bool few = p->n_tokens <= 64;
    dim3 grid((n + 127) / 128, few ? p->n_tokens : (p->n_tokens + 7) / 8);
    if (grid.y > 65535) return SPITE_UNSUPPORTED;
    auto decays = few ? channel_decays_kernel<1> : channel_decays_kernel<8>;
    SPITE_LAUNCH(decays, grid, 128, 0, st, a, a_stride, a2, b, (float*)p->w, p->w_stride, p->n_tokens, n, rank, 1.f / tau);
    if (cudaGetLastError() != cudaSuccess) return SPITE_LAUNCH_FAILED;
    if (chunks) return key_decay_in_chunks<false, PER_CHANNEL>(*p, scratch, n_chunks, min_tokens, st);
    return choose_scan<PER_CHANNEL>(*p, st);
}
SPITE_API int spite_gated_linear_scan(const ScanParams* p, const float* a, long long a_stride, const float* a2, const float* b,
                                      int rank, float tau, void* stream) {
    return gated_linear_scan(p, a, a_stride, a2, b, rank, tau, false, nullptr, 0, 0, stream);
}
SPITE_API int spite_gated_linear_scan_chunked(const ScanParams* p, const float* a, long long a_stride, const float* a2, const float* b, int rank,
                                              float tau, void* scratch, int n_chunks, int min_tokens, void* stream) {
    return gated_linear_scan(p, a, a_stride, a2, b, rank, tau, true, scratch, n_chunks, min_tokens, stream);
}
