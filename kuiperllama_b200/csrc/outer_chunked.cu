// The recurrence of outer_recurrence.cu over whole prompts, in chunks of 32 tokens on the tensor cores:
//
//   S_t = diag(a_t) S_(t-1) + (c_t k_t) v_t^T,     y_t = S_t^T (q_scale q_t) + D v_t
//
// A token i of a chunk that starts from S_in has, with A(j, i) the product of the decays a_(j+1) .. a_i and E_i the one from the chunk's
// first token on,
//
//   y_i = S_in^T E_i q_i + sum over j <= i of (q_i . A(j, i) c_j k_j) v_j,      S_out = E_end S_in + sum over j of (A(j, end) c_j k_j) v_j^T
//
// Walked token by token this is a chain of dependent steps (a prompt of 2,222 tokens took 584 us, 0.42 instructions a cycle); in chunks it is
// three products of matrices a chunk, and the chain is 32 times shorter.  Two launches:
//
//   oc_group_kernel, oc_row_kernel   a CTA per (chunk, unit, sequence): everything that does not depend on S.  One decay per head (MODE 0):
//       k and q of a group as they enter the products, their products q_i . k_j, and per head the decays' products A.  One decay per
//       row of S (MODE 1): q and k with their decays, and the weighted products.
//   oc_walk_kernel   a CTA per (32 columns of S, head, sequence) walks the chunks.  A warp holds 16 columns by half of the rows of S^T in
//       float32 accumulators, whose layout is also that of a product's first operand: S never leaves the registers.
//
// Nothing is rounded to 16 bits.  A 32-bit number enters a product as the sum of three bfloat16 numbers (24 bits of mantissa); of two such
// operands the six products down to 2^-16 of the leading one are added, smallest first; a bfloat16 operand enters as it is.  Products of
// decays are made as products (no logarithms, no quotients), at most 32 factors long, in 64 bits (those of 16 neighbouring tokens in 32, as the walk does).
// A chunk in which something is not finite, larger than OC_MOST, or whose decays leave [0, 1], is walked token by token (oc_tokens), so that
// infinities and NaN stay where they arise: a masked product would pass them on to the tokens before them.
//
// What bounds it: a chunk's chain of instructions (2.3 us where the products of mma.m16n8k16, six where there was one, take 0.9 of the tensor
// cores' time: 38 % busy, 0.33 instructions a cycle and scheduler).  One prompt of 2,048 tokens, us token by token / in chunks: 64 heads of
// 128 x 64 (state-space) 416 / 151, 16 heads of 64 x 128 with a decay per row (gated linear attention) 374 / 114; three prompts of 446, 1,333 and
// 2,222 tokens of the former 585 / 266.  Error against 64 bits, one sequence of 500 tokens with decays as such layers have: y 7.5e-8 / 7.0e-8 and
// 1.08e-7 / 8.8e-8, S 8.4e-8 / 6.7e-8 and 8.3e-8 / 5.3e-8.  With a decay per row and decays far from one (sigmoid(z) ** (1 / tau), tau 1 to 4) y 0.91 to
// 0.998 of the walk's, and S, which the walk then rounds once and this three times, 3.0e-8 to 4.6e-8 / 4.7e-8 to 6.1e-8: within one unit of 2^-24 either way.
//
// ExiledOfCode/KuiperLLama has no recurrent mixer (its mixer is mha_kernel.cu:61,74-106).
#include "pieces.cuh"

namespace kl {

constexpr int OC = 32;                     // tokens of a chunk: two blocks of 16
constexpr int OC_COLS = 32;                // columns of S of a CTA
constexpr int OC_THREADS = 128;            // of the CTAs that prepare
constexpr int OC_WARPS = 8;                // of the walk: two blocks of 16 columns by four quarters of the rows of S
constexpr int OC_FAC = 20;                 // factors of a (token, head): 16 of its block's products, E, from the block's start, to the block's end, to the chunk's end
constexpr int OC_MS = OC + 4;              // row stride of the products q . k in shared memory
constexpr float OC_MOST = 1048576.f;       // 2^20: what 2^20 chunks of such q, k, c and v add to S stays below 2^85, and its products with q below 2^112
constexpr float OC_MOST_S = OC_MOST * OC_MOST * OC_MOST;      // of S at the start

struct OuterChunkArgs {
    const void* q; long long ld_q; const void* k; long long ld_k; const void* v; long long ld_v;   // group g at column g * N, head h of v at h * P
    const float* a; long long ld_a; const float* c; long long ld_c; const float* skip;
    float* state; long long ld_state;
    float* y; long long ld_y;
    const int* cu_tokens; const int* seq_slots;
    // What the walk copies to shared memory as it lies, a piece per (chunk, unit); units: groups, or heads with a decay per row.  Rows of tokens
    // that a chunk does not have are zeros.
    unsigned char* qp;                     // [chunks, units]: q in three pieces [3][OC][NP]; with a decay per row then the weighted products of the
                                           //     chunk's tokens in three pieces [3][OC][OC], the chunk's decays [NP], and whether the chunk goes token by token [4]
    unsigned char* kp;                     // [chunks, units]: k in three pieces [3][OC][NP]
    float* prod;                           // [chunks, groups] (one decay per head): the products of the chunk's tokens [OC][OC_MS] and whether it goes token by token [4]
    float* fac;                            // [chunks, heads] (one decay per head): [OC][OC_FAC] and the same [4]
    int heads, groups, N, P;
    int chunk0, span;                      // the chunks of every sequence that this launch works: `span` of them from chunk0 on (0: all)
    float q_scale;
};

// The place of a chunk that starts at row `row0` of sequence s among all chunks: a sequence's chunks follow one another, and no two share one.
__device__ __forceinline__ size_t oc_entry(int row0, int s) { return (size_t)(row0 / OC + s); }
// The same in a portion of `span` chunks a sequence, from chunk0 on: first row of the portion's first chunk, and its place.
__device__ __forceinline__ int oc_first(const OuterChunkArgs& A, int s) { return A.cu_tokens[s] + A.chunk0 * OC; }
__device__ __forceinline__ size_t oc_entry0(const OuterChunkArgs& A, int s) { return A.span > 0 ? (size_t)s * A.span : oc_entry(A.cu_tokens[s], s); }
constexpr int OC_PROD = OC * OC_MS + 4, OC_FACS = OC * OC_FAC + 4;             // floats of a piece of `prod` and of `fac`
template <int NP> constexpr int oc_k_bytes() { return 3 * OC * NP * 2; }
template <int NP, int MODE> constexpr int oc_q_bytes() { return oc_k_bytes<NP>() + (MODE == 1 ? 3 * OC * OC * 2 + NP * 4 + 256 : 0); }

__device__ __forceinline__ bool oc_wild(float x) { return !(fabsf(x) <= OC_MOST); }      // too large, infinite or NaN

// ------------------------------------------------------------------------------------------ what does not depend on S
// One decay per head.  blockIdx.y < groups: k and q of a group in three pieces, and the products q_scale q_i . k_j of the chunk's tokens.
// Beyond: the products of decays of four heads, a warp each, a token a lane.
template <int NP>
__global__ void __launch_bounds__(OC_THREADS)
oc_group_kernel(const OuterChunkArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(256) unsigned char oc_raw[];
    const int s = blockIdx.z, ch = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = oc_first(A, s) + ch * OC, live = min(OC, A.cu_tokens[s + 1] - row0);
    if (live <= 0) return;
    const size_t entry = oc_entry0(A, s) + ch;
    if ((int)blockIdx.y >= A.groups) {
        const int h = (blockIdx.y - A.groups) * 4 + warp;
        if (h >= A.heads) return;
        const size_t row = (size_t)(row0 + min(lane, live - 1));
        const float a = lane < live ? A.a[row * A.ld_a + h] : 1.f;
        const float c = lane >= live ? 0.f : A.c != nullptr ? A.c[row * A.ld_c + h] : 1.f;
        const bool wild = oc_wild(c) || !(a >= 0.f && a <= 1.f);
        const unsigned any = __ballot_sync(0xffffffffu, wild);
        float* fac = A.fac + (entry * A.heads + h) * OC_FACS;
        if (lane == 0) reinterpret_cast<int*>(fac + OC * OC_FAC)[0] = any != 0;
        const int t = lane & 15;
        // (running products in 64 bits: a product of 32 decays is rounded once)
        double pre = a, suf = a;                           // from the block's start to here; from here to its end
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, pre, o, 16), down = __shfl_down_sync(0xffffffffu, suf, o, 16);
            if (t >= o) pre *= up;
            if (t + o < 16) suf *= down;
        }
        suf = __shfl_down_sync(0xffffffffu, suf, 1, 16);   // without this token's own
        if (t == 15) suf = 1.0;
        const double first = __shfl_sync(0xffffffffu, pre, 15), second = __shfl_sync(0xffffffffu, pre, 31);
        float d[16];                                       // c_j times the decays from the block's token j (exclusive) to here
        double r = 1.0;
#pragma unroll
        for (int j = 15; j >= 0; --j) {
            const float aj = __shfl_sync(0xffffffffu, a, j, 16), cj = __shfl_sync(0xffffffffu, c, j, 16);
            d[j] = j <= t ? (float)(cj * r) : 0.f;
            r = j <= t ? r * aj : 1.0;
        }
        float4* f = reinterpret_cast<float4*>(fac + lane * OC_FAC);
        const bool in = lane < live;
#pragma unroll
        for (int j = 0; j < 16; j += 4) f[j / 4] = in ? make_float4(d[j], d[j + 1], d[j + 2], d[j + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
        f[4] = in ? make_float4((float)(lane < 16 ? pre : first * pre), (float)pre, (float)(c * suf), (float)(c * (lane < 16 ? suf * second : suf))) : make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const int g = blockIdx.y, N = A.N;
    bf16* Qs = reinterpret_cast<bf16*>(oc_raw);            // [3][OC][NP]
    bf16* Ks = Qs + 3 * OC * NP;
    bf16* qp = reinterpret_cast<bf16*>(A.qp + (entry * A.groups + g) * oc_q_bytes<NP, 0>());
    float* prod = A.prod + (entry * A.groups + g) * OC_PROD;
    bf16* kp = reinterpret_cast<bf16*>(A.kp + (entry * A.groups + g) * oc_k_bytes<NP>());
    constexpr int TURNS = OC * NP / 8 / OC_THREADS;
    bool wild = false;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
        float4 x[TURNS][2];
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int e = threadIdx.x + OC_THREADS * i, r = e / (NP / 8), p = e % (NP / 8);
            const float* src = which ? (const float*)A.k + (size_t)(row0 + r) * A.ld_k : (const float*)A.q + (size_t)(row0 + r) * A.ld_q;
            const bool in = r < live && p * 8 < N;         // N is a multiple of eight
            src += (size_t)g * N + p * 8;
            x[i][0] = in ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
            x[i][1] = in ? *reinterpret_cast<const float4*>(src + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int e = threadIdx.x + OC_THREADS * i, r = e / (NP / 8), p = e % (NP / 8);
            uint32_t w[3][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float4 v = x[i][u];
                wild = wild || oc_wild(v.x) || oc_wild(v.y) || oc_wild(v.z) || oc_wild(v.w);
                pc_split(v.x, v.y, w[0][2 * u], w[1][2 * u], w[2][2 * u]);
                pc_split(v.z, v.w, w[0][2 * u + 1], w[1][2 * u + 1], w[2][2 * u + 1]);
            }
            bf16* tile = which ? Ks : Qs;
            bf16* out = which ? kp : qp;
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                const uint4 v = make_uint4(w[y][0], w[y][1], w[y][2], w[y][3]);
                *reinterpret_cast<uint4*>(tile + y * OC * NP + pc_at<NP>(r, p)) = v;
                *reinterpret_cast<uint4*>(out + y * OC * NP + pc_at<NP>(r, p)) = v;
            }
        }
    }
    const int any = __syncthreads_or(wild);
    if (threadIdx.x == 0) reinterpret_cast<int*>(prod + OC * OC_MS)[0] = any;
    const int rt = warp & 1, ct = warp >> 1;               // 16 tokens by 16 tokens a warp; nothing above the diagonal is asked for
    float d[2][4], small[2][4];
    pc_zero<2>(d);
    pc_zero<2>(small);
    if (ct <= rt) {
#pragma unroll 2
        for (int ks = 0; ks < NP / 16; ++ks) {
            uint32_t a[3][4], b[3][2][2];
            float main[2][4];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                pc_ldm4(smem_u32(Qs + i * OC * NP + pc_at<NP>(rt * 16 + (lane & 15), ks * 2 + (lane >> 4))), a[i]);
                pc_rows<NP, 2>(Ks + i * OC * NP, ct * 16, ks * 2, lane, b[i]);
            }
            pc_mma33<2, false>(main, small, a, b);
            pc_add<2>(d, main);
        }
        pc_add<2>(d, small);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float* o = prod + (rt * 16 + (lane >> 2) + 8 * i) * OC_MS + ct * 16 + 2 * (lane & 3);
        *reinterpret_cast<float2*>(o) = make_float2(A.q_scale * d[0][2 * i], A.q_scale * d[0][2 * i + 1]);
        *reinterpret_cast<float2*>(o + 8) = make_float2(A.q_scale * d[1][2 * i], A.q_scale * d[1][2 * i + 1]);
    }
}

// A decay per row of S, bfloat16 q and k: a CTA per (chunk, head, sequence).  q times E and c k times its decays to the chunk's end, in three
// pieces; the weighted products of the chunk's tokens: between the two blocks of 16 tokens as a product of q times the decays from
// the block's start and k times those to its block's end, inside a block term by term with a running product.
template <int NP>
__global__ void __launch_bounds__(OC_THREADS)
oc_row_kernel(const OuterChunkArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int RS = NP + 4;                             // row stride: rows four banks apart
    extern __shared__ __align__(256) unsigned char oc_raw[];
    float* as = reinterpret_cast<float*>(oc_raw);          // [OC][RS]: decays, then c k with them
    float* qs = as + OC * RS;                              // q_scale q
    float* ks = qs + OC * RS;                              // c k
    double* pre = reinterpret_cast<double*>(ks + OC * RS); // [2][NP]: the blocks' whole products
    float* ms = reinterpret_cast<float*>(pre + 2 * NP);    // [OC][OC_MS]: the weighted products
    const int s = blockIdx.z, h = blockIdx.y, ch = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = A.N;
    const int row0 = oc_first(A, s) + ch * OC, live = min(OC, A.cu_tokens[s + 1] - row0);
    if (live <= 0) return;
    const int g = h / (A.heads / A.groups);
    const size_t entry = oc_entry0(A, s) + ch;
    unsigned char* qm = A.qp + (entry * A.heads + h) * oc_q_bytes<NP, 1>();
    bf16* kp = reinterpret_cast<bf16*>(A.kp + (entry * A.heads + h) * oc_k_bytes<NP>());
    bool wild = false;
    for (int idx = threadIdx.x; idx < OC * NP / 8; idx += OC_THREADS) {
        const int r = idx / (NP / 8), p = idx % (NP / 8);
        const size_t row = (size_t)(row0 + r);
        float x[8], y[8], d[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) { x[u] = 0.f; y[u] = 0.f; d[u] = 1.f; }
        if (r < live && p * 8 < N) {
            const float c = A.c != nullptr ? A.c[row * A.ld_c + h] : 1.f;
            const uint4 qv = *reinterpret_cast<const uint4*>((const bf16*)A.q + row * A.ld_q + (size_t)g * N + p * 8);
            const uint4 kv = *reinterpret_cast<const uint4*>((const bf16*)A.k + row * A.ld_k + (size_t)g * N + p * 8);
            const float4* av = reinterpret_cast<const float4*>(A.a + row * A.ld_a + (size_t)h * N + p * 8);
            const float4 a0 = av[0], a1 = av[1];
            d[0] = a0.x; d[1] = a0.y; d[2] = a0.z; d[3] = a0.w; d[4] = a1.x; d[5] = a1.y; d[6] = a1.z; d[7] = a1.w;
            const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w}, kw[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x[2 * u] = A.q_scale * __uint_as_float(qw[u] << 16); x[2 * u + 1] = A.q_scale * __uint_as_float(qw[u] & 0xffff0000u);
                y[2 * u] = c * __uint_as_float(kw[u] << 16); y[2 * u + 1] = c * __uint_as_float(kw[u] & 0xffff0000u);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) wild = wild || oc_wild(x[u]) || oc_wild(y[u]) || !(d[u] >= 0.f && d[u] <= 1.f);
        }
#pragma unroll
        for (int u = 0; u < 8; u += 4) {
            *reinterpret_cast<float4*>(as + r * RS + p * 8 + u) = make_float4(d[u], d[u + 1], d[u + 2], d[u + 3]);
            *reinterpret_cast<float4*>(qs + r * RS + p * 8 + u) = make_float4(x[u], x[u + 1], x[u + 2], x[u + 3]);
            *reinterpret_cast<float4*>(ks + r * RS + p * 8 + u) = make_float4(y[u], y[u + 1], y[u + 2], y[u + 3]);
        }
    }
    const int any = __syncthreads_or(wild);
    if (threadIdx.x == 0) reinterpret_cast<int*>(qm + oc_q_bytes<NP, 1>() - 16)[0] = any;
    // inside a block: token j's c k, decayed from token to token, by the q of the tokens from j on.  Four lanes share the sum, each in eight parts
    // (short chains of additions: with one of 32 y's error was up to 1.2 times the walk's).
    {
        constexpr int E = NP / 4;                          // elements a lane: fours, sixteen apart
        const int b0 = (threadIdx.x >> 6) * 16, j = (threadIdx.x >> 2) & 15, part = threadIdx.x & 3;
        float r[E];
#pragma unroll
        for (int e = 0; e < E; e += 4) {
            const float4 x = *reinterpret_cast<const float4*>(ks + (b0 + j) * RS + e * 4 + part * 4);
            r[e] = x.x; r[e + 1] = x.y; r[e + 2] = x.z; r[e + 3] = x.w;
        }
        for (int i = 0; i < 16; ++i) {
            const bool on = i >= j;
            float parts[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < E; e += 4) {
                float* sums = parts + (e & 4);
                const float4 x = *reinterpret_cast<const float4*>(qs + (b0 + i) * RS + e * 4 + part * 4);
                const float4 d = *reinterpret_cast<const float4*>(as + (b0 + i) * RS + e * 4 + part * 4);
                if (i > j) { r[e] *= d.x; r[e + 1] *= d.y; r[e + 2] *= d.z; r[e + 3] *= d.w; }
                sums[0] = fmaf(x.x, r[e], sums[0]); sums[1] = fmaf(x.y, r[e + 1], sums[1]); sums[2] = fmaf(x.z, r[e + 2], sums[2]); sums[3] = fmaf(x.w, r[e + 3], sums[3]);
            }
            float sum = ((parts[0] + parts[1]) + (parts[2] + parts[3])) + ((parts[4] + parts[5]) + (parts[6] + parts[7]));
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if (part == 0) {
                float* o = ms + (b0 + i) * OC_MS;
                o[b0 + j] = on ? sum : 0.f;
                o[(b0 ^ 16) + j] = 0.f;                    // (between the blocks: below)
            }
        }
    }
    // the blocks' whole products of decays, in 64 bits as all of these products: what leaves here is rounded once
    for (int idx = threadIdx.x; idx < 2 * NP; idx += OC_THREADS) {
        const int b = idx / NP, n = idx % NP;
        double r = 1.0;
#pragma unroll
        for (int t = 0; t < 16; ++t) r *= as[(b * 16 + t) * RS + n];
        pre[idx] = r;
    }
    __syncthreads();
    // Along the tokens of a block: q times the decays from the block's start, in `as` k times those to its end.  For the walk, which counts from the chunk's start
    // and to its end, the other block's decays belong to q of the second block and to k of the first: those go to `ks`.
    for (int idx = threadIdx.x; idx < 2 * NP; idx += OC_THREADS) {
        const int b = idx / NP, n = idx % NP;
        const double other = pre[(b ^ 1) * NP + n];
        float whole[16];
        const double before = b ? other : 1.0, behind = b ? 1.0 : other;
        double r = 1.0, f = 1.0;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const int at = (b * 16 + t) * RS + n;
            r *= as[at];
            const double q = qs[at] * r;
            qs[at] = (float)q;
            whole[t] = (float)(q * before);
        }
#pragma unroll
        for (int t = 15; t >= 0; --t) {
            const int at = (b * 16 + t) * RS + n;
            const float a = as[at];
            const double k = ks[at] * f;
            as[at] = (float)k;
            ks[at] = b ? whole[t] : (float)(k * behind);
            f *= a;
        }
    }
    __syncthreads();
    if (warp == 0 && live > 16) {                          // between the blocks
        float d[2][4], small[2][4];
        pc_zero<2>(d);
        pc_zero<2>(small);
        const int r = lane >> 2, kc = 2 * (lane & 3);
#pragma unroll 2
        for (int kk = 0; kk < NP / 16; ++kk) {
            uint32_t a[3][4], b[3][2][2];
            float main[2][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x = *reinterpret_cast<const float2*>(qs + (16 + r + 8 * (e & 1)) * RS + kk * 16 + kc + 8 * (e >> 1));
                pc_split(x.x, x.y, a[0][e], a[1][e], a[2][e]);
                const float2 z = *reinterpret_cast<const float2*>(as + (r + 8 * (e & 1)) * RS + kk * 16 + kc + 8 * (e >> 1));
                pc_split(z.x, z.y, b[0][e & 1][e >> 1], b[1][e & 1][e >> 1], b[2][e & 1][e >> 1]);
            }
            pc_mma33<2, false>(main, small, a, b);
            pc_add<2>(d, main);
        }
        pc_add<2>(d, small);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float* o = ms + (16 + r + 8 * i) * OC_MS + kc;
            *reinterpret_cast<float2*>(o) = make_float2(d[0][2 * i], d[0][2 * i + 1]);
            *reinterpret_cast<float2*>(o + 8) = make_float2(d[1][2 * i], d[1][2 * i + 1]);
        }
    }
    // q and k for the walk in pieces (rows past the end are zeros: so are their k and q)
    for (int idx = threadIdx.x; idx < OC * NP / 8 * 2; idx += OC_THREADS) {
        const int which = idx / (OC * NP / 8), e = idx % (OC * NP / 8), r = e / (NP / 8), p = e % (NP / 8);
        const float* src = ((r < 16) == (which != 0) ? ks : which ? as : qs) + r * RS + p * 8;
        bf16* out = which ? kp : reinterpret_cast<bf16*>(qm);
        uint32_t w[3][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            pc_split(src[2 * u], src[2 * u + 1], w[0][u], w[1][u], w[2][u]);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(out + i * OC * NP + pc_at<NP>(r, p)) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
    }
    float* alpha = reinterpret_cast<float*>(qm + 3 * OC * NP * 2 + 3 * OC * OC * 2);
    for (int n = threadIdx.x; n < NP; n += OC_THREADS) alpha[n] = (float)(pre[n] * pre[NP + n]);
    __syncthreads();
    {                                                      // the weighted products, eight of a row a thread
        const int i = threadIdx.x >> 2, q4 = threadIdx.x & 3;
        const float* m = ms + i * OC_MS + q4 * 8;
        bf16* out = reinterpret_cast<bf16*>(qm + 3 * OC * NP * 2);
        uint32_t w[3][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) pc_split(m[2 * u], m[2 * u + 1], w[0][u], w[1][u], w[2][u]);
#pragma unroll
        for (int x = 0; x < 3; ++x) *reinterpret_cast<uint4*>(out + x * OC * OC + pc_at<OC>(i, q4)) = make_uint4(w[x][0], w[x][1], w[x][2], w[x][3]);
    }
}

// ------------------------------------------------------------------------------------------ the walk over the chunks
// Shared memory of the walk, in bytes, two of each: q (and what comes with it), k, the products and the factors (one decay per head), the weights in
// three pieces, v in three pieces (as it is and with the decays to the chunk's end), the quarters' shares of y; then four barriers.
template <int NP, int MODE>
struct OcWalk {
    static constexpr int Q_BYTES = oc_q_bytes<NP, MODE>(), K_BYTES = oc_k_bytes<NP>(), F_BYTES = MODE == 0 ? (OC_PROD + OC_FACS) * 4 : 0,
                         M_BYTES = MODE == 0 ? 3 * OC * OC * 2 : 0, V_BYTES = 2 * (MODE == 0 ? 2 * 2 * 3 : 2) * 512, Y_BYTES = OC_WARPS * 4 * 512;
    static constexpr int K = 2 * Q_BYTES, F = K + 2 * K_BYTES, M = F + 2 * F_BYTES, V = M + 2 * M_BYTES, Y = V + 2 * V_BYTES, BARS = Y + 2 * Y_BYTES, BYTES = BARS + 32;
    static_assert(Q_BYTES % 256 == 0 && K_BYTES % 256 == 0 && F_BYTES % 16 == 0 && BYTES <= 227 * 1024, "oc_walk_kernel: rows of 16-byte pieces, shared memory");
    static_assert(Y_BYTES >= NP * OC_COLS * 4 && V_BYTES >= OC_WARPS * 32 * 4, "what oc_tokens borrows");
};
template <int MODE> struct OcIn { typedef float type; };
template <> struct OcIn<1> { typedef bf16 type; };

// A chunk's tokens one by one, S [NP][OC_COLS] in shared memory, a thread per column and eighth of the rows.
template <int NP, int MODE>
__device__ __noinline__ void oc_tokens(const OuterChunkArgs& A, float* S, float* part, int row0, int live, int h, int g) {
    typedef typename OcIn<MODE>::type TI;
    constexpr int PARTS = OC_WARPS * 32 / OC_COLS;
    const int p = threadIdx.x % OC_COLS, mine = threadIdx.x / OC_COLS, col = blockIdx.x * OC_COLS + p;
    for (int t = 0; t < live; ++t) {
        const size_t row = (size_t)(row0 + t);
        const float c = A.c != nullptr ? A.c[row * A.ld_c + h] : 1.f;
        const float x = col < A.P ? to_f32(((const TI*)A.v)[row * A.ld_v + (size_t)h * A.P + col]) : 0.f;
        float sum = 0.f;
        for (int n = mine * (NP / PARTS); n < min(A.N, (mine + 1) * (NP / PARTS)); ++n) {
            const float a = MODE == 1 ? A.a[row * A.ld_a + (size_t)h * A.N + n] : A.a[row * A.ld_a + h];
            const float v = fmaf(a, S[n * OC_COLS + p], to_f32(((const TI*)A.k)[row * A.ld_k + (size_t)g * A.N + n]) * (c * x));
            S[n * OC_COLS + p] = v;
            sum = fmaf(v, to_f32(((const TI*)A.q)[row * A.ld_q + (size_t)g * A.N + n]), sum);
        }
        part[threadIdx.x] = sum;
        __syncthreads();
        if (mine == 0 && col < A.P) {
            float y = part[p];
            for (int i = 1; i < PARTS; ++i) y += part[p + i * OC_COLS];
            A.y[row * A.ld_y + (size_t)h * A.P + col] = A.skip != nullptr ? fmaf(A.skip[h], x, A.q_scale * y) : A.q_scale * y;
        }
        __syncthreads();
    }
}

// What bounds a walk is how long a chunk takes one CTA: its warps' chains of dependent instructions, and the 16-byte pieces that the products read
// from shared memory (a tile of 16 columns uses a piece of q or k twice).  So a chunk's work is cut over eight warps and little is done twice: a
// warp holds 16 columns of S by a quarter of its rows in registers, brings 8 tokens of v in pieces to shared memory for all, and finishes the y
// of 8 tokens from the four quarters' shares.  Between two barriers lie the products of a chunk, the preparation of the next one and the end of the
// one before, none of which waits for another; everything in shared memory is there twice, and one thread copies the operands of the next
// chunk as they lie (bulk copies).
// PART: of a portion of the step's chunks (A.span); without it the walk is 1.5 % faster than with a test.
template <int NP, int MODE, bool PART>
__global__ void __launch_bounds__(OC_WARPS * 32, NP == 64 && MODE == 1 ? 2 : 1)
oc_walk_kernel(const OuterChunkArgs A) {
    pdl_wait();
    typedef OcWalk<NP, MODE> L;
    constexpr int NQ = NP / 4, KT = NQ / 16, ST = NQ / 8;  // rows of S a warp holds, as steps of a product and as tiles
    extern __shared__ __align__(256) unsigned char oc_raw[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(oc_raw + L::BARS);            // q and k of either buffer, products and factors of either buffer
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pw = warp & 1, nq = warp >> 1;
    // The longest sequences start first (prompts of 446, 1,333 and 2,222 tokens, 64 heads of 128 x 64: 266 us, 292 in the order they come): with up to 32 of them, a lane each.
    int s = blockIdx.z;
    if (gridDim.z > 1 && gridDim.z <= 32) {
        const int mine = lane < gridDim.z ? A.cu_tokens[lane + 1] - A.cu_tokens[lane] : -1;
        int longer = 0;
        for (int i = 0; i < (int)gridDim.z; ++i) {
            const int len = __shfl_sync(0xffffffffu, mine, i);
            longer += len > mine || (len == mine && i < lane);
        }
        s = __ffs(__ballot_sync(0xffffffffu, lane < gridDim.z && longer == (int)blockIdx.z)) - 1;
    }
    const int first = PART ? oc_first(A, s) : A.cu_tokens[s], rest = A.cu_tokens[s + 1] - first, n_new = PART ? min(rest, A.span * OC) : rest, h = blockIdx.y;
    if (n_new <= 0) return;
    const int chunks = (n_new + OC - 1) / OC;
    const int r = lane >> 2, kc = 2 * (lane & 3);
    const int N = A.N, P = A.P, g = h / (A.heads / A.groups), units = MODE == 1 ? A.heads : A.groups, unit = MODE == 1 ? h : g;
    const int p0 = blockIdx.x * OC_COLS + pw * 16;
    const bool on = p0 < P;                                // P is a multiple of 16
    const size_t entry0 = PART ? (size_t)s * A.span : oc_entry(first, s);
    float* S_slot = A.state + (size_t)A.seq_slots[s] * A.ld_state + (size_t)h * N * P;
    const float skip = A.skip != nullptr ? A.skip[h] : 0.f;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mbar_init(bars + i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    auto copy_operands = [&](int c) {
        if (threadIdx.x == 0 && c < chunks) {
            const int b = c & 1;
            mbar_expect_tx(bars + b, L::Q_BYTES + L::K_BYTES);
            pc_bulk(oc_raw + b * L::Q_BYTES, A.qp + ((entry0 + c) * units + unit) * L::Q_BYTES, L::Q_BYTES, bars + b);
            pc_bulk(oc_raw + L::K + b * L::K_BYTES, A.kp + ((entry0 + c) * units + unit) * L::K_BYTES, L::K_BYTES, bars + b);
        }
    };
    auto copy_factors = [&](int c) {
        if (MODE == 0 && threadIdx.x == 0 && c < chunks) {
            const int b = c & 1;
            mbar_expect_tx(bars + 2 + b, L::F_BYTES);
            pc_bulk(oc_raw + L::F + b * L::F_BYTES, A.prod + ((entry0 + c) * A.groups + g) * OC_PROD, OC_PROD * 4, bars + 2 + b);
            pc_bulk(oc_raw + L::F + b * L::F_BYTES + OC_PROD * 4, A.fac + ((entry0 + c) * A.heads + h) * OC_FACS, OC_FACS * 4, bars + 2 + b);
        }
    };
    // A copy of this CTA's own always arrives; the limit is there so that no wait is without one (a chunk whose wait ran out goes token by token).
    auto wait = [&](int which, int c) {
        bool here = false;
        for (uint32_t i = 0; i < SPIN_LIMIT && !here; ++i) here = mbar_try_wait(bars + which + (c & 1), (c >> 1) & 1);
        return here;
    };
    // v of the warp's 8 tokens: tokens nq * 8 + kc, + 1 of columns r and r + 8
    const size_t v_at = (size_t)(first + nq * 8 + kc) * A.ld_v + (size_t)h * P + p0 + r;
    auto load_v = [&](int c, float2 (&x)[2]) {
        const int live = on ? n_new - c * OC - nq * 8 - kc : 0;
        const typename OcIn<MODE>::type* v = (const typename OcIn<MODE>::type*)A.v + v_at + (size_t)c * OC * A.ld_v;
#pragma unroll
        for (int e = 0; e < 2; ++e) x[e] = make_float2(live > 0 ? to_f32(v[8 * e]) : 0.f, live > 1 ? to_f32(v[A.ld_v + 8 * e]) : 0.f);
    };
    // v^T as the first operand of products over tokens: a lane's words of a step of 16 tokens; MODE 0: [as it is, decayed][step][piece], 1: [step]
    auto words_of_v = [&](int b) { return reinterpret_cast<uint4*>(oc_raw + L::V + b * L::V_BYTES) + pw * (MODE == 0 ? 12 : 2) * 32 + lane; };
    auto shares = [&](int b) { return reinterpret_cast<float4*>(oc_raw + L::Y + b * L::Y_BYTES) + lane; };     // [quarter][columns][tokens / 8]
    float S[ST][4];                                        // S^T: columns r, r + 8 of S by rows kc, kc + 1 of each tile
    auto large = [&]() {                                   // something in S is larger than OC_MOST_S, infinite or NaN
        unsigned most = 0;
#pragma unroll
        for (int n = 0; n < ST; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) most = max(most, __float_as_uint(S[n][e]) & 0x7fffffffu);
        return most > __float_as_uint(OC_MOST_S);
    };
    // chunk c, whose factors have arrived: the weights of its tokens, v in pieces.  `next` keeps what is needed later.
    struct Kept { float from[2], alpha; } now = {{1.f, 1.f}, 1.f}, next = now;             // E of two tokens, the chunk's decay (one per head)
    auto prepare = [&](int c, const float2 (&x)[2]) {
        const int b = c & 1;
        uint32_t* mine = reinterpret_cast<uint32_t*>(words_of_v(b) + (nq >> 1) * (MODE == 0 ? 3 : 1) * 32) + 2 * (nq & 1);
        bool wild = oc_wild(x[0].x) || oc_wild(x[0].y) || oc_wild(x[1].x) || oc_wild(x[1].y);
        if constexpr (MODE == 0) {
            const float* Ms = reinterpret_cast<const float*>(oc_raw + L::F + b * L::F_BYTES);
            const float* Fs = Ms + OC_PROD;
            wild = wild || (reinterpret_cast<const int*>(Ms + OC * OC_MS)[0] | reinterpret_cast<const int*>(Fs + OC * OC_FAC)[0]) != 0;
            bf16* Mp = reinterpret_cast<bf16*>(oc_raw + L::M + b * L::M_BYTES);
            const int i = threadIdx.x >> 3, j0 = (threadIdx.x & 7) * 4;                    // four of a row a thread
            float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j0 < 16 || i >= 16) {
                const float4 y = *reinterpret_cast<const float4*>(Ms + i * OC_MS + j0), f = *reinterpret_cast<const float4*>(Fs + i * OC_FAC + (j0 & 15));
                const float from = Fs[i * OC_FAC + 17], *to = Fs + j0 * OC_FAC + 18;
                const bool near = (i >= 16) == (j0 >= 16);                                 // in one block
                w.x = y.x * (near ? f.x : from * to[0]);
                w.y = y.y * (near ? f.y : from * to[OC_FAC]);
                w.z = y.z * (near ? f.z : from * to[2 * OC_FAC]);
                w.w = y.w * (near ? f.w : from * to[3 * OC_FAC]);
            }
            uint32_t pc[3][2];
            pc_split(w.x, w.y, pc[0][0], pc[1][0], pc[2][0]);
            pc_split(w.z, w.w, pc[0][1], pc[1][1], pc[2][1]);
#pragma unroll
            for (int y = 0; y < 3; ++y) *reinterpret_cast<uint2*>(Mp + y * OC * OC + pc_at<OC>(i, j0 >> 3) + (j0 & 7)) = make_uint2(pc[y][0], pc[y][1]);
            const float* f = Fs + (nq * 8 + kc) * OC_FAC;
            const float to0 = f[19], to1 = f[OC_FAC + 19];
            next.from[0] = A.q_scale * f[16];
            next.from[1] = A.q_scale * f[OC_FAC + 16];
            next.alpha = Fs[(min(OC, n_new - c * OC) - 1) * OC_FAC + 16];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t p[3], d[3];
                pc_split(x[e].x, x[e].y, p[0], p[1], p[2]);
                pc_split(x[e].x * to0, x[e].y * to1, d[0], d[1], d[2]);
#pragma unroll
                for (int y = 0; y < 3; ++y) { mine[y * 128 + e] = p[y]; mine[768 + y * 128 + e] = d[y]; }
            }
        } else {
#pragma unroll
            for (int e = 0; e < 2; ++e) mine[e] = (__float_as_uint(x[e].x) >> 16) | (__float_as_uint(x[e].y) & 0xffff0000u);
        }
        return wild;
    };
    // the y of the warp's tokens of chunk c, whose shares are whole: `mine` is the skip and what the chunk's own tokens give
    auto finish = [&](int c, const float (&mine)[4], const float (&from)[2]) {
        const float4* share = shares(c & 1) + (pw * 4 + nq) * 32;
        float4 far = share[0];
#pragma unroll
        for (int w = 1; w < 4; ++w) {
            const float4 more = share[w * 8 * 32];
            far.x += more.x; far.y += more.y; far.z += more.z; far.w += more.w;
        }
        float* y = A.y + (size_t)(first + c * OC + nq * 8 + kc) * A.ld_y + (size_t)h * P + p0 + r;
        const int left = on ? n_new - c * OC - nq * 8 - kc : 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float f = e == 0 ? far.x : e == 1 ? far.y : e == 2 ? far.z : far.w;
            if ((e & 1) < left) y[(e & 1) * A.ld_y + 8 * (e >> 1)] = MODE == 0 ? fmaf(f, from[e & 1], mine[e]) : f + mine[e];
        }
    };

    float2 x_now[2], x_next[2], x_later[2];
    copy_operands(0);
    copy_factors(0);
    copy_factors(1);
    load_v(0, x_now);
    load_v(1, x_next);
#pragma unroll
    for (int n = 0; n < ST; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = nq * NQ + n * 8 + kc + (e & 1);
            S[n][e] = on && row < N ? S_slot[(size_t)row * P + p0 + r + 8 * (e >> 1)] : 0.f;
        }
    bool wild_state = large(), wild = MODE == 0 && !wait(2, 0);
    wild = prepare(0, x_now) || wild;
    // where a lane reads pieces of q (rows of tokens) and k (rows of tokens, turned): the piece of a step by exclusive or
    const uint32_t q_lane = smem_u32(oc_raw) + ((lane & 7) + ((lane >> 4) << 3)) * NP * 2 + ((((lane >> 3) & 1) ^ (lane & 7)) << 4);
    const uint32_t k_lane = smem_u32(oc_raw + L::K) + (lane & 15) * NP * 2 + (((lane >> 4) ^ (lane & 7)) << 4);
    const uint32_t m_lane = smem_u32(oc_raw + (MODE == 1 ? oc_k_bytes<NP>() : L::M)) + pc_at<OC>(nq * 8 + (lane & 7), lane >> 3) * 2;
    float mine[4], from[2] = {1.f, 1.f};                   // of the chunk before
    bool left = false;                                     // its y is to be finished

    for (int c = 0; c < chunks; ++c) {
        const int b = c & 1;
        wild = !wait(0, c) || wild || wild_state;
        if (MODE == 0 && c + 1 < chunks) wild = !wait(2, c + 1) || wild;
        if constexpr (MODE == 1) wild = wild || *reinterpret_cast<const int*>(oc_raw + (b + 1) * L::Q_BYTES - 16) != 0;
        const int slow = __syncthreads_or(wild);           // what was prepared and shared is there; everyone is done with the other buffers
        copy_operands(c + 1);
        copy_factors(c + 2);
        load_v(c + 2, x_later);
        if (left) finish(c - 1, mine, from);
        left = !slow;
        now = next;
        wild = c + 1 < chunks && prepare(c + 1, x_next);
        if (slow) {
            float* St = reinterpret_cast<float*>(oc_raw + L::Y + b * L::Y_BYTES);          // [NP][OC_COLS]
#pragma unroll
            for (int n = 0; n < ST; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) St[(nq * NQ + n * 8 + kc + (e & 1)) * OC_COLS + pw * 16 + r + 8 * (e >> 1)] = S[n][e];
            __syncthreads();
            oc_tokens<NP, MODE>(A, St, reinterpret_cast<float*>(oc_raw + L::V + b * L::V_BYTES), first + c * OC, min(OC, n_new - c * OC), h, g);
#pragma unroll
            for (int n = 0; n < ST; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] = St[(nq * NQ + n * 8 + kc + (e & 1)) * OC_COLS + pw * 16 + r + 8 * (e >> 1)];
            wild_state = large();
        } else {
            // S^T q: this quarter of the rows, all 32 tokens
            {
                float Y[4][4], small[4][4];
#pragma unroll
                for (int ks = 0; ks < KT; ++ks) {
                    uint32_t a[3][4], f[3][4][2];
                    float more[4][4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) pc_split(S[2 * ks + (e >> 1)][2 * (e & 1)], S[2 * ks + (e >> 1)][2 * (e & 1) + 1], a[0][e], a[1][e], a[2][e]);
                    const uint32_t at = (q_lane + b * L::Q_BYTES) ^ ((nq * KT + ks) << 5);
#pragma unroll
                    for (int x = 0; x < 3; ++x)
#pragma unroll
                        for (int n = 0; n < 4; n += 2) {
                            uint32_t w[4];
                            pc_ldm4(at + (x * OC + n * 8) * NP * 2, w);
                            f[x][n][0] = w[0]; f[x][n][1] = w[1]; f[x][n + 1][0] = w[2]; f[x][n + 1][1] = w[3];
                        }
                    if (ks == 0) {
                        pc_mma33<4, true>(Y, small, a, f);
                    } else {
                        pc_mma33<4, false>(more, small, a, f);
                        pc_add<4>(Y, more);
                    }
                }
                float4* share = shares(b) + warp * 4 * 32;
#pragma unroll
                for (int n = 0; n < 4; ++n)
                    share[n * 32] = make_float4(Y[n][0] + small[n][0], Y[n][1] + small[n][1], Y[n][2] + small[n][2], Y[n][3] + small[n][3]);
            }
            // S^T = its decay + v^T (decayed c k)
            {
                const uint4* V = words_of_v(b) + (MODE == 0 ? 6 * 32 : 0);
                float main[ST][4], small[ST][4];
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    uint32_t f[3][ST][2];
#pragma unroll
                    for (int n = 0; n < ST; n += 2) {
                        const uint32_t at = (k_lane + b * L::K_BYTES) ^ ((nq * ST + n) << 4);
#pragma unroll
                        for (int x = 0; x < 3; ++x) {
                            uint32_t w[4];
                            pc_ldm4t(at + (x * OC + ks * 16) * NP * 2, w);
                            f[x][n][0] = w[0]; f[x][n][1] = w[1]; f[x][n + 1][0] = w[2]; f[x][n + 1][1] = w[3];
                        }
                    }
                    float more[ST][4];
                    if constexpr (MODE == 1) {
                        const uint4 w = V[ks * 32];
                        const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int n = 0; n < ST; ++n)
                            if (ks == 0) pc_mma0(small[n], a, f[2][n][0], f[2][n][1]); else pc_mma(small[n], a, f[2][n][0], f[2][n][1]);
#pragma unroll
                        for (int n = 0; n < ST; ++n) pc_mma(small[n], a, f[1][n][0], f[1][n][1]);
#pragma unroll
                        for (int n = 0; n < ST; ++n) pc_mma0(ks ? more[n] : main[n], a, f[0][n][0], f[0][n][1]);
                    } else {
                        uint32_t a[3][4];
#pragma unroll
                        for (int x = 0; x < 3; ++x) {
                            const uint4 w = V[(ks * 3 + x) * 32];
                            a[x][0] = w.x; a[x][1] = w.y; a[x][2] = w.z; a[x][3] = w.w;
                        }
                        if (ks == 0) pc_mma33<ST, true>(main, small, a, f); else pc_mma33<ST, false>(more, small, a, f);
                    }
                    if (ks) pc_add<ST>(main, more);
                }
#pragma unroll
                for (int n = 0; n < ST; ++n) {
                    float2 alpha = make_float2(now.alpha, now.alpha);
                    if constexpr (MODE == 1)
                        alpha = *reinterpret_cast<const float2*>(oc_raw + b * L::Q_BYTES + oc_k_bytes<NP>() + 3 * OC * OC * 2 + (nq * NQ + n * 8 + kc) * 4);
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[n][e] = fmaf((e & 1) ? alpha.y : alpha.x, S[n][e], main[n][e] + small[n][e]);
                }
            }
            // what the chunk's own tokens give the warp's, and the skip
            {
                const uint4* V = words_of_v(b);
                const uint32_t at = m_lane + b * (MODE == 1 ? L::Q_BYTES : L::M_BYTES);
                uint32_t m[3][4];
#pragma unroll
                for (int x = 0; x < 3; ++x) pc_ldm4(at + x * OC * OC * 2, m[x]);
                float own[4], lo[4], hi[4] = {0.f, 0.f, 0.f, 0.f}, more[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    if (ks == 0 || nq >= 2) {
                        uint32_t a[MODE == 1 ? 1 : 3][4];
#pragma unroll
                        for (int x = 0; x < (MODE == 1 ? 1 : 3); ++x) {
                            const uint4 w = V[(MODE == 1 ? ks : ks * 3 + x) * 32];
                            a[x][0] = w.x; a[x][1] = w.y; a[x][2] = w.z; a[x][3] = w.w;
                        }
                        if constexpr (MODE == 1) {
                            if (ks == 0) pc_mma0(lo, a[0], m[2][0], m[2][1]); else pc_mma(lo, a[0], m[2][2], m[2][3]);
                            pc_mma(hi, a[0], m[1][2 * ks], m[1][2 * ks + 1]);
                            pc_mma0(ks ? more : own, a[0], m[0][2 * ks], m[0][2 * ks + 1]);
                        } else {
                            if (ks == 0) pc_mma0(lo, a[2], m[0][0], m[0][1]); else pc_mma(lo, a[2], m[0][2], m[0][3]);
                            pc_mma(hi, a[1], m[0][2 * ks], m[0][2 * ks + 1]);
                            pc_mma0(ks ? more : own, a[0], m[0][2 * ks], m[0][2 * ks + 1]);
                            pc_mma(lo, a[1], m[1][2 * ks], m[1][2 * ks + 1]);
                            pc_mma(hi, a[0], m[1][2 * ks], m[1][2 * ks + 1]);
                            pc_mma(lo, a[0], m[2][2 * ks], m[2][2 * ks + 1]);
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) mine[e] = fmaf(skip, (e & 1) ? x_now[e >> 1].y : x_now[e >> 1].x, (own[e] + more[e]) + (lo[e] + hi[e]));
                from[0] = now.from[0];
                from[1] = now.from[1];
            }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) { x_now[e] = x_next[e]; x_next[e] = x_later[e]; }
    }
    pdl_launch_dependents();
    __syncthreads();
    if (left) finish(chunks - 1, mine, from);
    if (!on) return;
#pragma unroll
    for (int n = 0; n < ST; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = nq * NQ + n * 8 + kc + (e & 1);
            if (row < N) S_slot[(size_t)row * P + p0 + r + 8 * (e >> 1)] = S[n][e];
        }
}

template <int NP, int MODE>
static int launch_outer_chunked(const OuterChunkArgs& A, int chunks, int n_seqs, cudaStream_t stream) {
    const int pre = MODE == 0 ? 2 * 3 * OC * NP * 2 : (3 * OC * (NP + 4) + 4 * NP + OC * OC_MS) * 4;
    if constexpr (MODE == 0) {
        KL_CUDA(cudaFuncSetAttribute(oc_group_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, pre));
        launch_kernel(oc_group_kernel<NP>, dim3(chunks, A.groups + (A.heads + 3) / 4, n_seqs), OC_THREADS, pre, stream, A);
    } else {
        KL_CUDA(cudaFuncSetAttribute(oc_row_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, pre));
        launch_kernel(oc_row_kernel<NP>, dim3(chunks, A.heads, n_seqs), OC_THREADS, pre, stream, A);
    }
    KL_LAUNCH_CHECK();
    constexpr int smem = OcWalk<NP, MODE>::BYTES;
    const auto walk = A.span > 0 ? oc_walk_kernel<NP, MODE, true> : oc_walk_kernel<NP, MODE, false>;
    KL_CUDA(cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    launch_kernel_after(walk, dim3((A.P + OC_COLS - 1) / OC_COLS, A.heads, n_seqs), OC_WARPS * 32, smem, stream, A);
    KL_LAUNCH_CHECK();
    return KL_OK;
}

static long long oc_q(int N, int a_per_row) {
    return a_per_row ? (N <= 64 ? oc_q_bytes<64, 1>() : oc_q_bytes<128, 1>()) : (N <= 64 ? oc_q_bytes<64, 0>() : oc_q_bytes<128, 0>());
}
static long long oc_k(int N) { return N <= 64 ? oc_k_bytes<64>() : oc_k_bytes<128>(); }
static long long oc_round(long long bytes) { return (bytes + 255) / 256 * 256; }

// What a step's scratch holds: all chunks where they take up to `limit` bytes, else as many chunks of every sequence as that (one at least), and the step
// is worked in portions of so many.
struct OcPlan {
    long long units, entries, bytes;
    int chunks, span;                      // chunks of the longest sequence; of every sequence in a portion (0: all of them at once)
    OcPlan(int rows, int n_seqs, int max_new, int heads, int groups, int N, int a_per_row, long long limit) {
        units = a_per_row ? heads : groups;
        chunks = (max_new + OC - 1) / OC;
        const long long one = units * (oc_q(N, a_per_row) + oc_k(N)) + (a_per_row ? 0 : (long long)groups * OC_PROD * 4 + (long long)heads * OC_FACS * 4);
        entries = rows / OC + n_seqs + 1;
        span = 0;
        if (entries * one > limit) {
            const long long most = limit / one / n_seqs;
            span = most < 1 ? 1 : most < chunks ? (int)most : chunks;
            if ((long long)span * n_seqs < entries) entries = (long long)span * n_seqs;
            else span = 0;
        }
        bytes = oc_round(entries * units * oc_q(N, a_per_row)) + oc_round(entries * units * oc_k(N)) +
                (a_per_row ? 0 : oc_round(entries * groups * OC_PROD * 4) + oc_round(entries * heads * OC_FACS * 4));
    }
    int portions() const { return span > 0 ? (chunks + span - 1) / span : 1; }
};

}  // namespace kl

using namespace kl;

// 1 where the chunked form runs these sizes: float32 k, q and v with one decay per head, or bfloat16 ones with a decay per row of S; N a multiple of 8
// up to 128, P one of 16.
KL_API int kl_outer_chunked_fits(int n_seqs, int heads, int groups, int N, int P, int a_per_row, int in_dtype) {
    if (n_seqs <= 0 || heads <= 0 || groups <= 0 || heads % groups || heads + groups > 65535 || n_seqs > 65535) return 0;
    if (N <= 0 || N > 128 || N % 8 || P <= 0 || P % 16) return 0;
    return (in_dtype == KL_F32 && !a_per_row) || (in_dtype == KL_BF16 && a_per_row);
}
// Bytes of scratch that kl_outer_chunked needs, and in how many portions it works a step whose scratch keeps to `limit` bytes (two launches each).
KL_API long long kl_outer_chunked_scratch(int rows, int n_seqs, int max_new, int heads, int groups, int N, int a_per_row, long long limit) {
    return OcPlan(rows, n_seqs, max_new, heads, groups, N, a_per_row, limit).bytes;
}
KL_API int kl_outer_chunked_portions(int rows, int n_seqs, int max_new, int heads, int groups, int N, int a_per_row, long long limit) {
    return OcPlan(rows, n_seqs, max_new, heads, groups, N, a_per_row, limit).portions();
}

// q, k, v, a, c, skip, state and y as kl_outer_recurrence takes them (no normaliser); rows of k and q (and of a, with a decay per row) on
// 16-byte boundaries.  scratch: kl_outer_chunked_scratch bytes on a 16-byte boundary.
KL_API int kl_outer_chunked(const void* q, long long ld_q, const void* k, long long ld_k, const void* v, long long ld_v, const float* a, long long ld_a,
                            int a_per_row, const float* c, long long ld_c, const float* skip, float* state, long long ld_state, float* y,
                            long long ld_y, void* scratch, long long limit, const int* cu_tokens, const int* seq_slots, int rows, int n_seqs, int max_new,
                            int heads, int groups, int N, int P, float q_scale, int in_dtype, cudaStream_t stream) {
    if (rows <= 0 || n_seqs <= 0 || max_new <= 0) return KL_OK;
    if (!kl_outer_chunked_fits(n_seqs, heads, groups, N, P, a_per_row, in_dtype)) return KL_ERR_BAD_SIZE;
    const int w = in_dtype == KL_F32 ? 4 : 8;
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)scratch) & 15) || ld_q % w || ld_k % w || (a_per_row && (((uintptr_t)a & 15) || ld_a % 4))) return KL_ERR_BAD_ALIGN;
    const OcPlan plan(rows, n_seqs, max_new, heads, groups, N, a_per_row, limit);
    OuterChunkArgs A;
    A.q = q; A.ld_q = ld_q; A.k = k; A.ld_k = ld_k; A.v = v; A.ld_v = ld_v; A.a = a; A.ld_a = ld_a; A.c = c; A.ld_c = ld_c; A.skip = skip;
    A.state = state; A.ld_state = ld_state; A.y = y; A.ld_y = ld_y; A.cu_tokens = cu_tokens; A.seq_slots = seq_slots;
    A.heads = heads; A.groups = groups; A.N = N; A.P = P; A.q_scale = q_scale; A.span = plan.span;
    unsigned char* at = (unsigned char*)scratch;
    A.qp = at; at += oc_round(plan.entries * plan.units * oc_q(N, a_per_row));
    A.kp = at; at += oc_round(plan.entries * plan.units * oc_k(N));
    A.prod = a_per_row ? nullptr : (float*)at; at += a_per_row ? 0 : oc_round(plan.entries * groups * OC_PROD * 4);
    A.fac = a_per_row ? nullptr : (float*)at;
    for (int i = 0; i < plan.portions(); ++i) {            // (S goes from one portion to the next through the slot, as the 32-bit numbers that it is)
        A.chunk0 = i * plan.span;
        const int chunks = plan.span > 0 ? (plan.span < plan.chunks - A.chunk0 ? plan.span : plan.chunks - A.chunk0) : plan.chunks;
        const int rc = a_per_row ? (N <= 64 ? launch_outer_chunked<64, 1>(A, chunks, n_seqs, stream) : launch_outer_chunked<128, 1>(A, chunks, n_seqs, stream))
                                 : (N <= 64 ? launch_outer_chunked<64, 0>(A, chunks, n_seqs, stream) : launch_outer_chunked<128, 0>(A, chunks, n_seqs, stream));
        if (rc != KL_OK) return rc;
    }
    return KL_OK;
}
