// A linear recurrence whose state is a matrix per head, fed by outer products:
//
//   S_t = diag(a_t) S_(t-1) + (c_t k_t) v_t^T        S: [N, P] per head, float32, from the slot's state (zero in a fresh slot)
//   y_t = S_t^T q_t + D v_t                           y: [P] per head, float32
//
// a_t is one number per (token, head) (a state-space layer: exp(-exp(A_log) dt), with c_t = dt, k = B, q = C, v = x
// and the skip D) or one number per (token, head, row of S) (gated linear attention: c = 1, D = 0).  k and q may be
// shared by the heads of a group (head h reads group h / (heads / groups)).  Everything inside the recurrence is
// 32-bit; k, q and v are read in their own type (float32, or the compute dtype straight from a projection), q times
// q_scale.  A normaliser (a matrix memory with exponential gates, mLSTM) is one more column of S that is fed by c k alone:
//
//   n_t = diag(a_t) n_(t-1) + c_t k_t;     den_t = max(|n_t . q_t|, floor_t) + den_eps           [rows, heads]
//
//   outer_recurrence_kernel<TI, NPT>   a CTA per (sequence, head, block of columns of S).  A column of S is cut over
//       L lanes of one warp, lane l holding rows l, l + L, ... (NPT of them, in registers); tokens arrive in tiles
//       through shared memory; per token every thread decays and updates its rows, multiplies them by q and the
//       lanes' sums are added by shuffles.  Tokens are walked in order from the slot's state.
//   outer_recurrence_slab_kernel<TI, R, L, MODE>   the form that runs where the sizes allow: R x 2 of S per thread (see there).
//   outer_recurrence_few_kernel<TI, V, CL, T>   a step of at most eight tokens a sequence, bound by reading and writing S once:
//       neighbouring lanes hold neighbouring columns of a row, four or eight rows a thread on their way at a time.
//   Prompts of 64 tokens and more go in chunks on the tensor cores where the sizes allow (outer_chunked.cu).
//   decay_softplus_kernel     dt = softplus(raw + bias), a = exp(-exp(A_log) dt) per (token, head), 32-bit.
//   decay_lowrank_kernel      a = sigmoid(z)^(1 / tau) = exp(-softplus(-z) / tau), z = W2 r + b with r a short row per
//                             token (the first of two projections, made with the mixer's other projections), 32-bit.
//
// ExiledOfCode/KuiperLLama has no recurrent mixer (its mixer is mha_kernel.cu:61,74-106).
#include "common.cuh"

namespace kl {

constexpr int OR_THREADS = 512;          // the most threads of a CTA; a launch takes 128, 256 or 512
constexpr int OR_TILE = 32;           // tokens per shared-memory tile (the lane form)
constexpr int SLAB_WARPS = 10;         // warps an SM below which the slab form cuts S into smaller pieces

struct OuterArgs {
    const void* q; long long ld_q; int q_col;        // [rows, >= q_col + groups * N]
    const void* k; long long ld_k; int k_col;
    const void* v; long long ld_v; int v_col;        // [rows, >= v_col + heads * P]
    const float* a; long long ld_a;                  // [rows, heads] or [rows, heads * N]
    const float* c; long long ld_c;                  // [rows, heads] or null
    const float* skip;                               // [heads] or null
    float* state; long long ld_state;                // the slot's S at state + slot * ld_state, [heads, N, P]
    float* y; long long ld_y;                        // [rows, heads * P]
    const int* cu_tokens; const int* seq_slots;
    int heads, groups, N, P, L, a_per_row;
    int tile;                                        // tokens per shared-memory tile (the lane form; OR_TILE unless the rows are long)
    int vec_state;                                   // every row piece of four columns of S is 16-byte aligned
    int piece;                                       // elements of k, q and v to an asynchronous copy: four, what four bytes hold, or 0 (one by one)
    float q_scale;
    float* norm_state;                               // the slot's n at norm_state + slot * ld_state, [heads, N], or null
    const float* floor;                              // [rows, heads]
    float* den;                                      // [rows, heads]
    float den_eps;
};

__device__ __forceinline__ float or_den(const OuterArgs& A, size_t row, int h, float dot) {
    return fmaxf(fabsf(dot), A.floor[row * A.heads + h]) + A.den_eps;
}

template <typename TI, int NPT, bool NORM>
__global__ void __launch_bounds__(OR_THREADS, 1)
outer_recurrence_kernel(const OuterArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float sm[];
    const int s = blockIdx.z, h = blockIdx.y;
    const int row0 = A.cu_tokens[s], n_new = A.cu_tokens[s + 1] - row0;
    if (n_new <= 0) return;
    const int N = A.N, P = A.P, L = A.L;
    const int threads = blockDim.x;
    const int cols_per_cta = threads / L;
    const int lane = threadIdx.x % L;
    const int col = blockIdx.x * cols_per_cta + threadIdx.x / L;
    const bool live = col < P;
    const int g = h / (A.heads / A.groups);
    // shared: per tile token: k [N] (times c), q [N] (times q_scale), a [N or 1], v [cols_per_cta]
    const int a_len = A.a_per_row ? N : 1;
    const int per_tok = 2 * N + a_len + cols_per_cta;
    float* S_slot = A.state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N * P;
    float S[NPT];
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
        const int n = i * L + lane;
        S[i] = (live && n < N) ? S_slot[(size_t)n * P + col] : 0.f;
    }
    // the normaliser: the lanes of the first column of S carry it too
    const bool has_norm = NORM && blockIdx.x == 0 && threadIdx.x < 32;
    const bool in_norm = has_norm && threadIdx.x < L;
    float* n_slot = NORM ? A.norm_state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N : nullptr;
    float nS[NORM ? NPT : 1];
#pragma unroll
    for (int i = 0; i < (NORM ? NPT : 0); ++i) {
        const int n = i * L + lane;
        nS[i] = (in_norm && n < N) ? n_slot[n] : 0.f;
    }
    const TI* qp = (const TI*)A.q; const TI* kp = (const TI*)A.k; const TI* vp = (const TI*)A.v;
    const float skip = A.skip != nullptr ? A.skip[h] : 0.f;
    for (int t0 = 0; t0 < n_new; t0 += A.tile) {
        const int nt = min(A.tile, n_new - t0);
        __syncthreads();
        // the tile's k (times c), q (times q_scale), a and v, each in a loop of its own so that the loads of several
        // turns are in flight together
#pragma unroll 4
        for (int idx = threadIdx.x; idx < nt * N; idx += threads) {
            const int tt = idx / N, j = idx - tt * N;
            const size_t row = (size_t)(row0 + t0 + tt);
            float val = to_f32(kp[row * A.ld_k + A.k_col + (size_t)g * N + j]);
            if (A.c != nullptr) val *= A.c[row * A.ld_c + h];
            sm[tt * per_tok + j] = val;
        }
#pragma unroll 4
        for (int idx = threadIdx.x; idx < nt * N; idx += threads) {
            const int tt = idx / N, j = idx - tt * N;
            const size_t row = (size_t)(row0 + t0 + tt);
            sm[tt * per_tok + N + j] = to_f32(qp[row * A.ld_q + A.q_col + (size_t)g * N + j]) * A.q_scale;
        }
#pragma unroll 4
        for (int idx = threadIdx.x; idx < nt * a_len; idx += threads) {
            const int tt = idx / a_len, j = idx - tt * a_len;
            const size_t row = (size_t)(row0 + t0 + tt);
            sm[tt * per_tok + 2 * N + j] = A.a_per_row ? A.a[row * A.ld_a + (size_t)h * N + j] : A.a[row * A.ld_a + h];
        }
        for (int idx = threadIdx.x; idx < nt * cols_per_cta; idx += threads) {
            const int tt = idx / cols_per_cta, j = idx - tt * cols_per_cta;
            const size_t row = (size_t)(row0 + t0 + tt);
            const int cc = blockIdx.x * cols_per_cta + j;
            sm[tt * per_tok + 2 * N + a_len + j] = cc < P ? to_f32(vp[row * A.ld_v + A.v_col + (size_t)h * P + cc]) : 0.f;
        }
        __syncthreads();
        for (int tt = 0; tt < nt; ++tt) {
            const float* kk = sm + tt * per_tok;
            const float* qq = kk + N;
            const float* aa = qq + N;
            const float vv = aa[a_len + threadIdx.x / L];
            float acc = 0.f;
            if (A.a_per_row) {
#pragma unroll
                for (int i = 0; i < NPT; ++i) {
                    const int n = i * L + lane;
                    if (n < N) {
                        S[i] = fmaf(aa[n], S[i], kk[n] * vv);
                        acc = fmaf(S[i], qq[n], acc);
                    }
                }
            } else {
                const float a0 = aa[0];
#pragma unroll
                for (int i = 0; i < NPT; ++i) {
                    const int n = i * L + lane;
                    if (n < N) {
                        S[i] = fmaf(a0, S[i], kk[n] * vv);
                        acc = fmaf(S[i], qq[n], acc);
                    }
                }
            }
            for (int o = L >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0 && live) A.y[(size_t)(row0 + t0 + tt) * A.ld_y + (size_t)h * P + col] = fmaf(skip, vv, acc);
            if (NORM && has_norm) {
                float dot = 0.f;
#pragma unroll
                for (int i = 0; i < (NORM ? NPT : 0); ++i) {
                    const int n = i * L + lane;
                    if (in_norm && n < N) {
                        nS[i] = fmaf(A.a_per_row ? aa[n] : aa[0], nS[i], kk[n]);
                        dot = fmaf(nS[i], qq[n], dot);
                    }
                }
                for (int o = L >> 1; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                if (threadIdx.x == 0) A.den[(size_t)(row0 + t0 + tt) * A.heads + h] = or_den(A, (size_t)(row0 + t0 + tt), h, dot);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < (NORM ? NPT : 0); ++i) {
        const int n = i * L + lane;
        if (in_norm && n < N) n_slot[n] = nS[i];
    }
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
        const int n = i * L + lane;
        if (live && n < N) S_slot[(size_t)n * P + col] = S[i];
    }
}

__device__ __forceinline__ void or_ld4(const float* p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void or_ld4(const bf16* p, float (&x)[4]) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    x[0] = __uint_as_float(v.x << 16); x[1] = __uint_as_float(v.x & 0xffff0000u);
    x[2] = __uint_as_float(v.y << 16); x[3] = __uint_as_float(v.y & 0xffff0000u);
}

typedef unsigned long long f32x2;                              // two float32 numbers, one instruction for both
__device__ __forceinline__ f32x2 or_pair(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 or_unpair(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 or_fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 or_mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
template <int BYTES>
__device__ __forceinline__ void or_copy(void* dst, const void* src, bool live) {         // not live: the piece becomes zero, nothing is read
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(live ? BYTES : 0) : "memory");
}

// The same recurrence with R rows x 2 columns of S in a thread's registers, for prompts.  What bounds it is the chain of tokens: the
// arithmetic of a token is three multiply-adds an element, and a kernel that waits for shared memory, for shuffles and for the next
// tile of tokens between tokens spends most of its time there.  So: rows of S are packed in pairs (one instruction for two rows,
// and k, q and a of a pair come as they lie in shared memory), a thread reads four rows of k and q at once (L lanes read 16 L
// neighbouring bytes), four tokens are worked between reductions, whose eight sums the L lanes share out among themselves (seven
// shuffles for four tokens and two columns), and the next tile of tokens is copied while this one is worked.  One prompt of 2,048
// tokens, us with R x C of S per thread and a reduction per token and column / now: 64 heads of 128 x 64 (state-space) 1,043 / 405, 16
// heads of 64 x 128 with a decay per row (gated linear attention) 725 / 393; three prompts of 446, 1,333 and 2,222 tokens 1,668 / 585.
// Rows: lane rg holds rows 4 rg + 4 L i + (0..3), i < R / 4; rows from N to R L are zero and change nothing.
// MODE 0: one decay per head; 1: one per row of S; 2: one per head and the normaliser, which the first warp of the first columns carries.
constexpr int OSL_TOKENS = 4;             // tokens between reductions
constexpr int OSL_THREADS = 128;
// four neighbouring numbers as two pairs
__device__ __forceinline__ ulonglong2 or_quad(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ ulonglong2 or_quad(const bf16* p) {
    float x[4];
    or_ld4(p, x);
    return make_ulonglong2(or_pair(x[0], x[1]), or_pair(x[2], x[3]));
}
__device__ __forceinline__ float2 or_two(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 or_two(const bf16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }

template <typename TI, int R, int L, int MODE>
__global__ void __launch_bounds__(OSL_THREADS, 2)
outer_recurrence_slab_kernel(const OuterArgs A) {
    pdl_wait();
    constexpr int Np = R * L, H2 = R / 2, ES = sizeof(TI);
    constexpr int A_BYTES = MODE == 1 ? Np * 4 : 0;
    extern __shared__ __align__(16) unsigned char osl_smem[];
    const int s = blockIdx.z, h = blockIdx.y;
    const int row0 = A.cu_tokens[s], n_new = A.cu_tokens[s + 1] - row0;
    if (n_new <= 0) return;
    if (n_new <= 8) pdl_launch_dependents();                   // a few tokens; a walk over a prompt asks at its end, whatever its tile
    const int N = A.N, P = A.P, T = A.tile;
    const int threads = blockDim.x, lane = threadIdx.x & 31;
    const int rg = threadIdx.x % L, cg = threadIdx.x / L;      // the thread's lane along the rows, and its column pair in the CTA
    const int cols = threads / L * 2;                          // a multiple of four (the launch rounds its threads to that)
    const int col0 = blockIdx.x * cols + cg * 2;
    const bool live = col0 < P;                                // P is even
    const int g = h / (A.heads / A.groups);
    const int tok = (2 * Np * ES + A_BYTES + cols * ES + 15) / 16 * 16;       // bytes of a token: k, q, a, v
    const int scal = T * tok;                                  // behind them the tile's decays and factors c
    const int stage = (scal + 2 * T * 4 + 15) / 16 * 16;
    float* S_slot = A.state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N * P;

    // a thread copies the same four columns of every token of a tile
    auto copy_tile = [&](int t0, unsigned char* dst) {
        const int nt = min(T, n_new - t0);
        const size_t row = (size_t)(row0 + t0);
        const int kq = Np / 4, pieces = 2 * kq + (MODE == 1 ? kq : 0) + cols / 4;
        for (int j = threadIdx.x; j < pieces; j += threads) {
            const int which = j < kq ? 0 : j < 2 * kq ? 1 : (MODE == 1 && j < 3 * kq) ? 2 : 3;
            const int e = (j - (which == 3 && MODE != 1 ? 2 : which) * kq) * 4;
            const int c = which == 3 ? blockIdx.x * cols + e : e;                  // the element in its head's row
            const int n = min(4, (which == 3 ? P : N) - c);                        // elements that exist
            unsigned char* to = dst + (which == 0 ? e * ES : which == 1 ? (Np + e) * ES : which == 2 ? 2 * Np * ES + e * 4 : 2 * Np * ES + A_BYTES + e * ES);
            if (MODE == 1 && which == 2) {
                const float* src = A.a + row * A.ld_a + (size_t)h * N + c;
                for (int tt = 0; tt < T; ++tt, to += tok, src += A.ld_a) {
                    if (tt >= nt) *reinterpret_cast<float4*>(to) = make_float4(1.f, 1.f, 1.f, 1.f);      // a token past the end leaves S as it is
                    else if (A.piece == 4) or_copy<16>(to, n > 0 ? src : A.a, n > 0);
                    else
#pragma unroll
                        for (int u = 0; u < 4; ++u) or_copy<4>(to + 4 * u, u < n ? src + u : A.a, u < n);
                }
                continue;
            }
            const TI* base = (const TI*)(which == 0 ? A.k : which == 1 ? A.q : A.v);
            const long long ld = which == 0 ? A.ld_k : which == 1 ? A.ld_q : A.ld_v;
            const TI* src = base + row * ld + (which == 0 ? A.k_col + (size_t)g * N : which == 1 ? A.q_col + (size_t)g * N : A.v_col + (size_t)h * P) + c;
            if (A.piece == 4) {                                                    // N and P are multiples of four
                for (int tt = 0; tt < T; ++tt, to += tok, src += ld) {
                    const bool in = n > 0 && tt < nt;
                    or_copy<4 * ES>(to, in ? src : base, in);
                }
            } else if (A.piece > 0) {                                              // of what four bytes hold
                constexpr int W = 4 / ES;
                for (int tt = 0; tt < T; ++tt, to += tok, src += ld)
#pragma unroll
                    for (int u = 0; u < 4; u += W) {
                        const bool in = tt < nt && u < n;
                        or_copy<4>(to + u * ES, in ? src + u : base, in);
                    }
            } else {
                for (int t4 = 0; t4 < T; t4 += 4) {                                // T is a multiple of four: sixteen loads on their way together
                    TI x[4][4];
#pragma unroll
                    for (int tt = 0; tt < 4; ++tt)
#pragma unroll
                        for (int u = 0; u < 4; ++u) x[tt][u] = t4 + tt < nt && u < n ? src[(t4 + tt) * ld + u] : from_f32<TI>(0.f);
#pragma unroll
                    for (int tt = 0; tt < 4; ++tt)
#pragma unroll
                        for (int u = 0; u < 4; ++u) reinterpret_cast<TI*>(to + (t4 + tt) * tok)[u] = x[tt][u];
                }
            }
        }
        for (int t = threadIdx.x; t < 2 * T; t += threads) {
            const int tt = t < T ? t : t - T;
            float* to = reinterpret_cast<float*>(dst + scal) + t;
            const float* src = t < T ? (MODE != 1 ? A.a + (row + min(tt, nt - 1)) * A.ld_a + h : nullptr)
                                     : A.c != nullptr ? A.c + (row + min(tt, nt - 1)) * A.ld_c + h : nullptr;
            if (src != nullptr && tt < nt) or_copy<4>(to, src, true);
            else *to = 1.f;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    copy_tile(0, osl_smem);

    f32x2 S[H2][2];
#pragma unroll
    for (int i = 0; i < H2; ++i) {
        const int n = 4 * rg + 4 * L * (i / 2) + 2 * (i % 2);
#pragma unroll
        for (int j = 0; j < 2; ++j)
            S[i][j] = or_pair(live && n < N ? S_slot[(size_t)n * P + col0 + j] : 0.f, live && n + 1 < N ? S_slot[(size_t)(n + 1) * P + col0 + j] : 0.f);
    }
    const bool norm = MODE == 2 && blockIdx.x == 0 && threadIdx.x < 32;
    float* n_slot = MODE == 2 ? A.norm_state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N : nullptr;
    f32x2 nS[MODE == 2 ? H2 : 1];
    if constexpr (MODE == 2) {
#pragma unroll
        for (int i = 0; i < H2; ++i) {
            const int n = 4 * rg + 4 * L * (i / 2) + 2 * (i % 2);
            nS[i] = or_pair(norm && n < N ? n_slot[n] : 0.f, norm && n + 1 < N ? n_slot[n + 1] : 0.f);
        }
    }
    const float skip = A.skip != nullptr ? A.skip[h] : 0.f;

    int buf = 0;
    for (int t0 = 0; t0 < n_new; t0 += T, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                       // this tile is here, and everyone is done with the one before
        const unsigned char* tile = osl_smem + buf * stage;
        if (t0 + T < n_new) copy_tile(t0 + T, osl_smem + (buf ^ 1) * stage);
        const int nt = min(T, n_new - t0);
        const float* decay = reinterpret_cast<const float*>(tile + scal);
        const float* factor = decay + T;
        for (int tb = 0; tb < nt; tb += OSL_TOKENS) {
            float sums[OSL_TOKENS * 2];
            float dots[MODE == 2 ? OSL_TOKENS : 1];
#pragma unroll
            for (int u = 0; u < OSL_TOKENS; ++u) {             // T is a multiple of OSL_TOKENS; tokens past the end are zeros
                const unsigned char* at = tile + (tb + u) * tok;
                const TI* kk = reinterpret_cast<const TI*>(at) + 4 * rg;
                const float2 v = or_two(reinterpret_cast<const TI*>(at + 2 * Np * ES + A_BYTES) + 2 * cg);
                const float c = factor[tb + u], a0 = MODE == 1 ? 0.f : decay[tb + u];
                const f32x2 v0 = or_pair(c * v.x, c * v.x), v1 = or_pair(c * v.y, c * v.y), ad = or_pair(a0, a0), cd = or_pair(c, c);
                f32x2 y0[2] = {0, 0}, y1[2] = {0, 0}, dot = 0;
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    const ulonglong2 k4 = or_quad(kk + 4 * L * i), q4 = or_quad(kk + Np + 4 * L * i);
                    ulonglong2 a4 = make_ulonglong2(ad, ad);
                    if constexpr (MODE == 1) a4 = or_quad(reinterpret_cast<const float*>(at + 2 * Np * ES) + 4 * rg + 4 * L * i);
                    S[2 * i][0] = or_fma2(a4.x, S[2 * i][0], or_mul2(k4.x, v0));
                    S[2 * i][1] = or_fma2(a4.x, S[2 * i][1], or_mul2(k4.x, v1));
                    S[2 * i + 1][0] = or_fma2(a4.y, S[2 * i + 1][0], or_mul2(k4.y, v0));
                    S[2 * i + 1][1] = or_fma2(a4.y, S[2 * i + 1][1], or_mul2(k4.y, v1));
                    y0[0] = or_fma2(S[2 * i][0], q4.x, y0[0]);
                    y1[0] = or_fma2(S[2 * i][1], q4.x, y1[0]);
                    y0[1] = or_fma2(S[2 * i + 1][0], q4.y, y0[1]);
                    y1[1] = or_fma2(S[2 * i + 1][1], q4.y, y1[1]);
                    if constexpr (MODE == 2) {
                        if (norm) {
                            nS[2 * i] = or_fma2(ad, nS[2 * i], or_mul2(k4.x, cd));
                            nS[2 * i + 1] = or_fma2(ad, nS[2 * i + 1], or_mul2(k4.y, cd));
                            dot = or_fma2(nS[2 * i], q4.x, dot);
                            dot = or_fma2(nS[2 * i + 1], q4.y, dot);
                        }
                    }
                }
                const float2 s0 = or_unpair(y0[0]), s1 = or_unpair(y1[0]), s2 = or_unpair(y0[1]), s3 = or_unpair(y1[1]);
                sums[2 * u] = (s0.x + s0.y) + (s2.x + s2.y);
                sums[2 * u + 1] = (s1.x + s1.y) + (s3.x + s3.y);
                if constexpr (MODE == 2) { const float2 d = or_unpair(dot); dots[u] = d.x + d.y; }
            }
            // the lanes add each other's sums and keep a share: bit 0 of the lane the column, bits 1 and 2 the token (four lanes: two tokens each)
            int left = OSL_TOKENS * 2;
#pragma unroll
            for (int o = 1; o < L; o <<= 1) {
                if (left > 1) {
                    left >>= 1;
#pragma unroll
                    for (int j = 0; j < left; ++j) {
                        const float give = (lane & o) ? sums[2 * j] : sums[2 * j + 1], keep = (lane & o) ? sums[2 * j + 1] : sums[2 * j];
                        sums[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
                } else {
                    sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], o);
                }
            }
            constexpr int KEPT = L >= 8 ? 1 : 8 / L;
            if (live && rg < 8) {
#pragma unroll
                for (int j = 0; j < KEPT; ++j) {
                    const int idx = rg % 8 + j * (8 / KEPT), u = tb + idx / 2, cc = idx % 2;
                    if (u < nt) {
                        const float v = to_f32(reinterpret_cast<const TI*>(tile + u * tok + 2 * Np * ES + A_BYTES)[2 * cg + cc]);
                        A.y[(size_t)(row0 + t0 + u) * A.ld_y + (size_t)h * P + col0 + cc] = fmaf(skip, v, A.q_scale * sums[j]);
                    }
                }
            }
            if constexpr (MODE == 2) {
                if (norm) {
#pragma unroll
                    for (int u = 0; u < OSL_TOKENS; ++u) {
                        float d = dots[u];
#pragma unroll
                        for (int o = 1; o < L; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                        if (threadIdx.x == 0 && tb + u < nt) {
                            const size_t row = (size_t)(row0 + t0 + tb + u);
                            A.den[row * A.heads + h] = or_den(A, row, h, A.q_scale * d);
                        }
                    }
                }
            }
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < H2; ++i) {
        const int n = 4 * rg + 4 * L * (i / 2) + 2 * (i % 2);
        if constexpr (MODE == 2) {
            const float2 z = or_unpair(nS[i]);
            if (norm && cg == 0 && n < N) n_slot[n] = z.x;
            if (norm && cg == 0 && n + 1 < N) n_slot[n + 1] = z.y;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 x = or_unpair(S[i][j]);
            if (live && n < N) S_slot[(size_t)n * P + col0 + j] = x.x;
            if (live && n + 1 < N) S_slot[(size_t)(n + 1) * P + col0 + j] = x.y;
        }
    }
}

// At most T tokens per sequence (a step of single tokens: T = 1).  A CTA takes V CL columns of S of one (sequence, head); CL lanes hold
// V = 4 or 2 columns each and OS_THREADS / CL groups of lanes share the rows.  A row of S is read once, takes its tokens in order and is
// written once.  The slab form reads a column pair per lane, rows apart: 64 sequences of 2 tokens, us with slabs / here, 64 heads of
// 128 x 64 111 / 65, 8 heads of 256 x 256 with the normaliser 172 / 56; of 8 tokens 131 / 115 and 210 / 103.
constexpr int OS_THREADS = 256, OS_TOKENS = 8;
template <int V> struct OsCols;
template <> struct OsCols<4> { typedef float4 type; };
template <> struct OsCols<2> { typedef float2 type; };
template <typename TI, int V, int CL, int T>
__global__ void __launch_bounds__(OS_THREADS)
outer_recurrence_few_kernel(const OuterArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int RG = OS_THREADS / CL, U = T <= 2 ? 8 : 4;
    constexpr int PG = T > 1 && CL == 16 ? RG / 2 : RG;        // groups whose sums meet in shared memory (a warp's two add theirs first)
    extern __shared__ __align__(16) float sm[];
    __shared__ float scratch[33];
    const int s = blockIdx.z, h = blockIdx.y, N = A.N, P = A.P;
    const size_t row0 = (size_t)A.cu_tokens[s];
    const int nt = T == 1 ? min(1, A.cu_tokens[s + 1] - A.cu_tokens[s]) : min(T, A.cu_tokens[s + 1] - A.cu_tokens[s]);
    if (nt <= 0) return;
    const int g = h / (A.heads / A.groups);
    float4* kqa = reinterpret_cast<float4*>(sm);               // [T][N]: k times c, q times q_scale, a
    float* part = sm + 4 * T * N;                              // [PG][T][V CL]
    const int cl = threadIdx.x % CL, rg = threadIdx.x / CL;
    const int col = (blockIdx.x * CL + cl) * V;
    const bool live = col < P;                                 // P is a multiple of V
    typedef typename OsCols<V>::type Cols;
    float* S = A.state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N * P + col;
    for (int idx = threadIdx.x; idx < nt * N; idx += OS_THREADS) {
        const int t = T == 1 ? 0 : idx / N, n = idx - t * N;
        const size_t row = row0 + t;
        kqa[idx] = make_float4(to_f32(((const TI*)A.k)[row * A.ld_k + A.k_col + (size_t)g * N + n]) * (A.c != nullptr ? A.c[row * A.ld_c + h] : 1.f),
                               to_f32(((const TI*)A.q)[row * A.ld_q + A.q_col + (size_t)g * N + n]) * A.q_scale,
                               A.a_per_row ? A.a[row * A.ld_a + (size_t)h * N + n] : A.a[row * A.ld_a + h], 0.f);
    }
    float v[T][V], acc[T][V];
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int j = 0; j < V; ++j) {
            v[t][j] = live && t < nt ? to_f32(((const TI*)A.v)[(row0 + t) * A.ld_v + A.v_col + (size_t)h * P + col + j]) : 0.f;
            acc[t][j] = 0.f;
        }
    __syncthreads();
    for (int n0 = rg; n0 < N && live; n0 += RG * U) {
        float x[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int n = n0 + u * RG;
            const Cols w = n < N ? *reinterpret_cast<const Cols*>(S + (size_t)n * P) : Cols{};
#pragma unroll
            for (int j = 0; j < V; ++j) x[u][j] = reinterpret_cast<const float*>(&w)[j];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int n = n0 + u * RG;
            if (n >= N) break;
#pragma unroll
            for (int t = 0; t < T; ++t) {
                if (T > 1 && t >= nt) break;
                const float4 w = kqa[t * N + n];
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    x[u][j] = fmaf(w.z, x[u][j], w.x * v[t][j]);
                    acc[t][j] = fmaf(x[u][j], w.y, acc[t][j]);
                }
            }
            Cols w;
#pragma unroll
            for (int j = 0; j < V; ++j) reinterpret_cast<float*>(&w)[j] = x[u][j];
            *reinterpret_cast<Cols*>(S + (size_t)n * P) = w;
        }
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
        if constexpr (PG < RG) {
#pragma unroll
            for (int j = 0; j < V; ++j) acc[t][j] += __shfl_xor_sync(0xffffffffu, acc[t][j], 16);
        }
        if (PG == RG || rg % 2 == 0) {
#pragma unroll
            for (int j = 0; j < V; ++j) part[(size_t)((PG < RG ? rg / 2 : rg) * T + t) * V * CL + V * cl + j] = acc[t][j];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nt * V * CL; e += OS_THREADS) {
        const int t = e / (V * CL), at = blockIdx.x * V * CL + e % (V * CL);
        if (at >= P) continue;
        float y = 0.f;
#pragma unroll
        for (int r = 0; r < PG; ++r) y += part[(size_t)(r * T) * V * CL + e];
        const size_t row = row0 + t;
        if (A.skip != nullptr) y = fmaf(A.skip[h], to_f32(((const TI*)A.v)[row * A.ld_v + A.v_col + (size_t)h * P + at]), y);
        A.y[row * A.ld_y + (size_t)h * P + at] = y;
    }
    if (A.norm_state != nullptr && blockIdx.x == 0) {          // the normaliser: the first columns' CTA
        float* z = A.norm_state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N;
        float dot[T];
#pragma unroll
        for (int t = 0; t < T; ++t) dot[t] = 0.f;
        for (int n = threadIdx.x; n < N; n += OS_THREADS) {
            float x = z[n];
#pragma unroll
            for (int t = 0; t < T; ++t) {
                if (t >= nt) break;
                const float4 w = kqa[t * N + n];
                x = fmaf(w.z, x, w.x);
                dot[t] = fmaf(x, w.y, dot[t]);
            }
            z[n] = x;
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
            if (t >= nt) break;
            const float d = block_sum(dot[t], scratch);
            if (threadIdx.x == 0) A.den[(row0 + t) * A.heads + h] = or_den(A, row0 + t, h, d);
        }
    }
}

__global__ void decay_softplus_kernel(const void* __restrict__ raw, long long ld_raw, int col, int bf, const float* __restrict__ bias,
                                      const float* __restrict__ A_log, int rows, int heads, float* __restrict__ dt,
                                      float* __restrict__ a) {
    pdl_launch_dependents();
    pdl_wait();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= rows * heads) return;
    const int t = idx / heads, h = idx - t * heads;
    const size_t at = (size_t)t * ld_raw + col + h;
    float z = (bf ? __bfloat162float(((const bf16*)raw)[at]) : ((const float*)raw)[at]) + bias[h];
    const float d = z > 20.f ? z : log1pf(expf(z));
    dt[idx] = d;
    a[idx] = expf(-expf(A_log[h]) * d);
}

__device__ __forceinline__ float decay_of(float z, float inv_tau) {
    const float nz = -z;
    return expf(-(nz > 20.f ? nz : log1pf(expf(nz))) * inv_tau);
}

// a[t, c] = exp(-softplus(-z) / tau), z = b[c] + sum_r W2[c, r] * r1[t, r]
template <typename T>
__global__ void __launch_bounds__(256)
decay_lowrank_kernel(const T* __restrict__ r1, long long ld_r1, int col, int rank, const float* __restrict__ W2,
                     const float* __restrict__ b, float inv_tau, int rows, int channels, float* __restrict__ a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float row[];
    const int t = blockIdx.x;
    for (int r = threadIdx.x; r < rank; r += blockDim.x) row[r] = to_f32(r1[(size_t)t * ld_r1 + col + r]);
    __syncthreads();
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
        float z = 0.f;
        for (int r = 0; r < rank; ++r) z = fmaf(W2[(size_t)c * rank + r], row[r], z);
        z += b != nullptr ? b[c] : 0.f;
        a[(size_t)t * channels + c] = decay_of(z, inv_tau);
    }
}

// The same for short rows of 16: a thread keeps its channel's row of W2 in registers for `tile` tokens (a CTA per token read it again
// for every token: 66 us for 2,048 tokens of 1,024 channels, now 10).
constexpr int DL_RANK = 16, DL_TILE = 16;
template <typename T>
__global__ void __launch_bounds__(256)
decay_lowrank16_kernel(const T* __restrict__ r1, long long ld_r1, int col, const float* __restrict__ W2, const float* __restrict__ b,
                       float inv_tau, int rows, int channels, int tile, float* __restrict__ a) {
    pdl_launch_dependents();
    __shared__ __align__(16) float row[DL_TILE][DL_RANK];
    const int c = blockIdx.y * blockDim.x + threadIdx.x, t0 = blockIdx.x * tile, nt = min(tile, rows - t0);
    float w[DL_RANK], bias = 0.f;                              // weights: no kernel writes them
    if (c < channels) {
#pragma unroll
        for (int i = 0; i < DL_RANK; i += 4) *reinterpret_cast<float4*>(w + i) = *reinterpret_cast<const float4*>(W2 + (size_t)c * DL_RANK + i);
        if (b != nullptr) bias = b[c];
    }
    pdl_wait();
    for (int i = threadIdx.x; i < nt * DL_RANK; i += blockDim.x) row[i / DL_RANK][i % DL_RANK] = to_f32(r1[(size_t)(t0 + i / DL_RANK) * ld_r1 + col + i % DL_RANK]);
    __syncthreads();
    if (c >= channels) return;
    for (int t = 0; t < nt; ++t) {
        float z = 0.f;
#pragma unroll
        for (int i = 0; i < DL_RANK; i += 4) {
            const float4 r = *reinterpret_cast<const float4*>(&row[t][i]);
            z = fmaf(w[i], r.x, z); z = fmaf(w[i + 1], r.y, z); z = fmaf(w[i + 2], r.z, z); z = fmaf(w[i + 3], r.w, z);
        }
        a[(size_t)(t0 + t) * channels + c] = decay_of(z + bias, inv_tau);
    }
}

}  // namespace kl

using namespace kl;

// in_dtype: the type of q, k and v (KL_F32 or KL_BF16).  a_per_row != 0: a is [rows, heads * N].  norm_state (null: no normaliser)
// lies in the slot's state like `state`, ld_state apart; floor and den are float32 [rows, heads].
KL_API int kl_outer_recurrence(const void* q, long long ld_q, int q_col, const void* k, long long ld_k, int k_col, const void* v,
                               long long ld_v, int v_col, const float* a, long long ld_a, int a_per_row, const float* c,
                               long long ld_c, const float* skip, float* state, long long ld_state, float* y, long long ld_y,
                               const int* cu_tokens, const int* seq_slots, int n_seqs, int max_new, int heads, int groups, int N, int P,
                               float q_scale, float* norm_state, const float* floor, float* den, float den_eps, int in_dtype,
                               cudaStream_t stream) {
    if (n_seqs <= 0) return KL_OK;
    if (norm_state != nullptr && (floor == nullptr || den == nullptr)) return KL_ERR_BAD_SIZE;
    if (heads <= 0 || groups <= 0 || heads % groups || N <= 0 || P <= 0 || N > 1024) return KL_ERR_BAD_SIZE;
    if (in_dtype != KL_F32 && in_dtype != KL_BF16) return KL_ERR_BAD_DTYPE;
    int sms = 0, dev = 0;
    KL_CUDA(cudaGetDevice(&dev));
    KL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    OuterArgs A;
    A.q = q; A.ld_q = ld_q; A.q_col = q_col; A.k = k; A.ld_k = ld_k; A.k_col = k_col; A.v = v; A.ld_v = ld_v; A.v_col = v_col;
    A.a = a; A.ld_a = ld_a; A.c = c; A.ld_c = ld_c; A.skip = skip; A.state = state; A.ld_state = ld_state; A.y = y; A.ld_y = ld_y;
    A.cu_tokens = cu_tokens; A.seq_slots = seq_slots; A.heads = heads; A.groups = groups; A.N = N; A.P = P;
    A.a_per_row = a_per_row ? 1 : 0; A.q_scale = q_scale;
    A.norm_state = norm_state; A.floor = floor; A.den = den; A.den_eps = den_eps;
    A.vec_state = ((uintptr_t)state % 16 == 0 && ld_state % 4 == 0 && P % 4 == 0) ? 1 : 0;
    // a few tokens: S read and written once
    // (by slabs all the same: several tokens of narrow S, of which few lanes would have columns, 64 sequences of 4 heads of 16 x 8 by two 3.1 / 2.6
    // us; of few CTAs, one sequence of 4 heads of 500 x 64 by two 7.3 / 5.2; five and more tokens of small S, whose reading is not what takes
    // the time, 64 sequences of 32 heads of 64 x 64 by eight 32 / 28)
    const int vec = A.vec_state ? 4 : (uintptr_t)state % 8 == 0 && ld_state % 2 == 0 && P % 2 == 0 && P >= 16 ? 2 : 0;     // columns to a lane
    if (max_new <= OS_TOKENS && vec != 0 &&
        (max_new <= 1 || (P >= 8 * vec && (long long)((P + 63) / 64) * heads * n_seqs >= 16 && (max_new <= 4 || N * P > 4096)))) {
        // 64 columns a CTA where S has no more (128 leave half of the threads idle: 64 sequences of 64 heads of 128 x 64, 268 MB, 78 us
        // against 53) or where CTAs are few
        const bool narrow = P <= 64 || (long long)((P + 127) / 128) * heads * n_seqs < 2LL * sms;
        const int cols = vec == 2 ? 32 : narrow ? 64 : 128, T = max_new <= 1 && vec == 4 ? 1 : max_new <= 2 ? 2 : max_new <= 4 ? 4 : 8;
        const dim3 grid((P + cols - 1) / cols, heads, n_seqs);
        const size_t smem = (size_t)T * (4 * N + vec * OS_THREADS) * sizeof(float);
#define KL_FEW(TI, V, CL, T_)                                                                                        \
    do {                                                                                                            \
        if (smem > 47 * 1024)                                                                                       \
            KL_CUDA(cudaFuncSetAttribute(outer_recurrence_few_kernel<TI, V, CL, T_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        launch_kernel(outer_recurrence_few_kernel<TI, V, CL, T_>, grid, OS_THREADS, smem, stream, A);               \
    } while (0)
#define KL_FEW_T(TI, V, CL)                                                                                          \
    do {                                                                                                            \
        if (V == 4 && T == 1) KL_FEW(TI, 4, CL, 1); else if (T == 2) KL_FEW(TI, V, CL, 2); else if (T == 4) KL_FEW(TI, V, CL, 4); else KL_FEW(TI, V, CL, 8); \
    } while (0)
#define KL_FEW_V(TI)                                                                                                 \
    do {                                                                                                            \
        if (vec == 2) KL_FEW_T(TI, 2, 16); else if (narrow) KL_FEW_T(TI, 4, 16); else KL_FEW_T(TI, 4, 32);          \
    } while (0)
        if (in_dtype == KL_F32) KL_FEW_V(float); else KL_FEW_V(bf16);
#undef KL_FEW_V
#undef KL_FEW_T
#undef KL_FEW
        KL_LAUNCH_CHECK();
        return KL_OK;
    }
    // slabs of R x 2 in registers: the most rows a thread that still give the device SLAB_WARPS warps an SM, else the fewest.  us at R = 16 / 8
    // / 4: one prompt of 2,048 tokens, 64 heads of 128 x 64 (3.5 / 7 / 14 warps an SM) 478 / 427 / 405, 16 heads of 64 x 128 (1.7 / 3.5 / 6.9)
    // 620 / 528 / 398, eight prompts of 256 of the latter (14 / 28 / 55) 93 / 131 / 133.
    const int mode = norm_state != nullptr ? 2 : a_per_row ? 1 : 0;
    if (P % 2 == 0 && N <= 512 && !(mode == 2 && a_per_row)) {
        int R = 0, L = 0;
        for (int r = 16; r >= 4; r >>= 1) {
            int l = 4;
            while (l * r < N) l <<= 1;
            if (l > 32) continue;
            R = r; L = l;
            if (1LL * n_seqs * heads * l * (P / 2) / 32 >= (long long)SLAB_WARPS * sms) break;
        }
        const int pairs = P / 2, es = in_dtype == KL_F32 ? 4 : 2;
        // CTAs of 128 threads: a CTA's threads share the copies of a tile, two CTAs on an SM fill each other's waits
        const int fewest = 2 * L > 32 ? 2 * L : 32;            // whole warps and four columns of S at least
        // always a multiple of `fewest`, so that a CTA's columns are a multiple of four: v is copied in pieces of four columns
        int threads = (L * pairs + fewest - 1) / fewest * fewest;
        threads = threads > OSL_THREADS ? OSL_THREADS : threads;
        while (threads % (2 * fewest) == 0 && (long long)((pairs * L + threads - 1) / threads) * heads * n_seqs < sms) threads >>= 1;
        const int cols = threads / L * 2, Np = R * L, tok = (2 * Np * es + (mode == 1 ? Np * 4 : 0) + cols * es + 15) / 16 * 16;
        // the widest asynchronous copies that every row of k, q and v (and a) allows (8 heads of 20 x 50, bfloat16, 512 tokens: 213 us copied
        // element by element, 133 in pairs)
        auto whole = [&](int w) {
            auto rows = [&](const void* p, long long ld, int col) { return (uintptr_t)p % (w * es) == 0 && ld % w == 0 && col % w == 0; };
            return N % w == 0 && P % w == 0 && rows(q, ld_q, q_col) && rows(k, ld_k, k_col) && rows(v, ld_v, v_col);
        };
        A.piece = whole(4) && (!a_per_row || ((uintptr_t)a % 16 == 0 && ld_a % 4 == 0)) ? 4 : whole(4 / es) ? 4 / es : 0;
        A.tile = max_new <= 4 ? 4 : max_new <= 8 || Np > 256 ? 8 : 16;       // (a prompt of long rows of S: 8)
        A.L = L;
        const size_t smem = (size_t)2 * ((A.tile * tok + 2 * A.tile * 4 + 15) / 16 * 16);
        const dim3 grid((P + cols - 1) / cols, heads, n_seqs);
#define KL_SLAB(TI, R_, L_, M_)                                                                                      \
    do {                                                                                                            \
        if (smem > 48 * 1024)                                                                                       \
            KL_CUDA(cudaFuncSetAttribute(outer_recurrence_slab_kernel<TI, R_, L_, M_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        if (max_new > 8) launch_kernel_after(outer_recurrence_slab_kernel<TI, R_, L_, M_>, grid, threads, smem, stream, A); \
        else launch_kernel(outer_recurrence_slab_kernel<TI, R_, L_, M_>, grid, threads, smem, stream, A);           \
    } while (0)
#define KL_SLAB_M(TI, R_, L_)                                                                                        \
    do {                                                                                                            \
        if (mode == 0) KL_SLAB(TI, R_, L_, 0); else if (mode == 1) KL_SLAB(TI, R_, L_, 1); else KL_SLAB(TI, R_, L_, 2); \
    } while (0)
#define KL_SLAB_L(TI, R_)                                                                                            \
    do {                                                                                                            \
        if (L == 4) KL_SLAB_M(TI, R_, 4); else if (L == 8) KL_SLAB_M(TI, R_, 8); else if (L == 16) KL_SLAB_M(TI, R_, 16); else KL_SLAB_M(TI, R_, 32); \
    } while (0)
#define KL_SLAB_R(TI)                                                                                                \
    do {                                                                                                            \
        if (R == 16) KL_SLAB_L(TI, 16); else if (R == 8) KL_SLAB_L(TI, 8); else KL_SLAB_L(TI, 4);                   \
    } while (0)
        if (in_dtype == KL_F32) KL_SLAB_R(float); else KL_SLAB_R(bf16);
#undef KL_SLAB_R
#undef KL_SLAB_L
#undef KL_SLAB_M
#undef KL_SLAB
        KL_LAUNCH_CHECK();
        return KL_OK;
    }
    // any other size: a column of S over L lanes, rows of S in registers per thread at most 16 where 32 lanes allow it
    int L = 1;
    while (L < 32 && (N + L - 1) / L > 16) L <<= 1;
    // and more lanes (fewer rows per thread) while the launch would leave the SMs short of warps: a prompt of one sequence
    // is a chain of dependent steps per thread, and only other warps hide its latency
    long long warps = (long long)n_seqs * heads * P * L / 32;
    while (L < 32 && (N + L - 1) / L > 2 && warps < 24LL * sms) { L <<= 1; warps <<= 1; }
    const int npt = (N + L - 1) / L;
    A.L = L;
    // the largest CTA that still leaves two CTAs per SM (a CTA loads a tile of tokens, waits, and computes: another one
    // fills the wait), and no wider than the columns of S
    int threads = OR_THREADS;
    while (threads > 128 && (threads / 2 >= P * L || (long long)((P * L + threads - 1) / threads) * heads * n_seqs < 2LL * sms)) threads >>= 1;
    const int cols = threads / L;
    dim3 grid((P + cols - 1) / cols, heads, n_seqs);
    const size_t per_token = (size_t)(2 * N + (a_per_row ? N : 1) + cols) * sizeof(float);
    A.tile = OR_TILE;
    while (A.tile > 1 && A.tile * per_token > 200 * 1024) A.tile >>= 1;
    const size_t smem = A.tile * per_token;
    if (smem > 200 * 1024) return KL_ERR_BAD_SIZE;
#define KL_OR_N(TI, NPT, NM)                                                                                        \
    do {                                                                                                            \
        if (smem > 48 * 1024)                                                                                       \
            KL_CUDA(cudaFuncSetAttribute(outer_recurrence_kernel<TI, NPT, NM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        launch_kernel(outer_recurrence_kernel<TI, NPT, NM>, grid, threads, smem, stream, A);                        \
    } while (0)
#define KL_OR(TI, NPT)                                                                                              \
    do {                                                                                                            \
        if (norm_state != nullptr) KL_OR_N(TI, NPT, true); else KL_OR_N(TI, NPT, false);                            \
    } while (0)
#define KL_OR_BY_NPT(TI)                                                                                            \
    do {                                                                                                            \
        if (npt <= 2) KL_OR(TI, 2); else if (npt <= 4) KL_OR(TI, 4); else if (npt <= 8) KL_OR(TI, 8); else if (npt <= 16) KL_OR(TI, 16); else KL_OR(TI, 32); \
    } while (0)
    if (in_dtype == KL_F32) KL_OR_BY_NPT(float); else KL_OR_BY_NPT(bf16);
#undef KL_OR_BY_NPT
#undef KL_OR
#undef KL_OR_N
    KL_LAUNCH_CHECK();
    return KL_OK;
}

KL_API int kl_decay_softplus(const void* raw, long long ld_raw, int col, int dtype, const float* bias, const float* A_log, int rows,
                             int heads, float* dt, float* a, cudaStream_t stream) {
    if (rows <= 0 || heads <= 0) return KL_OK;
    if (dtype != KL_F32 && dtype != KL_BF16) return KL_ERR_BAD_DTYPE;
    const int total = rows * heads;
    launch_kernel(decay_softplus_kernel, (total + 255) / 256, 256, 0, stream, raw, ld_raw, col, (int)(dtype == KL_BF16), bias, A_log, rows,
                  heads, dt, a);
    KL_LAUNCH_CHECK();
    return KL_OK;
}

KL_API int kl_decay_lowrank(const void* r1, long long ld_r1, int col, int rank, const float* W2, const float* b, float tau, int rows,
                            int channels, float* a, int dtype, cudaStream_t stream) {
    if (rows <= 0 || channels <= 0) return KL_OK;
    if (rank <= 0 || rank > 4096 || !(tau > 0.f)) return KL_ERR_BAD_SIZE;
    int yblocks = (channels + 255) / 256;
    if (rank == DL_RANK && (uintptr_t)W2 % 16 == 0 && (dtype == KL_F32 || dtype == KL_BF16) && yblocks <= 65535) {
        int tile = DL_TILE;                                    // fewer tokens a CTA while the device has less than two CTAs an SM
        while (tile > 1 && (long long)((rows + tile - 1) / tile) * yblocks < 2LL * sm_count()) tile >>= 1;
        const dim3 g16((rows + tile - 1) / tile, yblocks);
        if (dtype == KL_F32)
            launch_kernel(decay_lowrank16_kernel<float>, g16, 256, 0, stream, (const float*)r1, ld_r1, col, W2, b, 1.0f / tau, rows, channels, tile, a);
        else
            launch_kernel(decay_lowrank16_kernel<bf16>, g16, 256, 0, stream, (const bf16*)r1, ld_r1, col, W2, b, 1.0f / tau, rows, channels, tile, a);
        KL_LAUNCH_CHECK();
        return KL_OK;
    }
    if (yblocks > 64) yblocks = 64;
    dim3 grid(rows, yblocks);
    if (dtype == KL_F32)
        launch_kernel(decay_lowrank_kernel<float>, grid, 256, rank * sizeof(float), stream, (const float*)r1, ld_r1, col, rank, W2, b, 1.0f / tau,
                      rows, channels, a);
    else if (dtype == KL_BF16)
        launch_kernel(decay_lowrank_kernel<bf16>, grid, 256, rank * sizeof(float), stream, (const bf16*)r1, ld_r1, col, rank, W2, b, 1.0f / tau,
                      rows, channels, a);
    else
        return KL_ERR_BAD_DTYPE;
    KL_LAUNCH_CHECK();
    return KL_OK;
}
