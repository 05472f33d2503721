// The gated delta rule of recurrent.cu over whole prompts, in chunks of 32 tokens on the tensor cores:
//
//   S <- g_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
//
// With A(s, t) the product of the decays g_(s+1) .. g_t, G_t the one from the chunk's first token on, and S the state before the chunk, the u of
// a chunk's tokens solve a triangular system (Yang et al., "Parallelizing Linear Transformers with the Delta Rule over Sequence Length",
// 2024):
//
//   u_t + sum over s < t of L_ts u_s = beta_t (v_t - G_t S^T k_t),   L_ts = beta_t A(s, t) (k_t . k_s)
//
// so with T = (I + L)^-1:  U = T (beta V) - W S,  W = T (beta G K);  o_t = G_t S^T q_t + sum over s <= t of A(s, t) (q_t . k_s) u_s;  and the
// chunk leaves  G_C S + sum over s of k_s A(s, C) u_s^T.  Walked token by token this is a chain of 2,048 dependent steps of 190 ns (389 us for a
// prompt of 2,048 tokens).  Three launches:
//
//   dc_prepare_kernel  the convolution, SiLU and unit lengths, beta and the decays: a warp per (8 tokens, key head or 128 channels of v), which
//                    keeps the taps before a token in registers.
//   dc_head_kernel   a CTA per (chunk, head, sequence): T by forward substitution, W, T (beta V), the weights A(s, t) (q_t . k_s); k and q in
//                    pieces once for the heads that share them.  Nothing here depends on S.
//   dc_walk_kernel   a CTA per (16 columns of S, head, sequence) walks the chunks.  A warp holds 16 rows of S for these columns in float32
//                    accumulators, which are also a first operand of products (pieces.cuh).
//
// Nothing is rounded to 16 bits: a 32-bit number enters a product as three bfloat16 numbers.  With unit keys and beta in [0, 1] no entry of
// T is above one.  A chunk in which something is not finite or too large, or whose beta or decays leave [0, 1], is walked token by token (dc_tokens).
// One prompt of 2,048 tokens with its preparation, us token by token / in chunks: 16 heads of 128 x 128 444 / 169, 8 420 / 142; error of y against 64
// bits, one sequence of 500 tokens, 2.4e-7 / 2.1e-7, of S 3.7e-7 / 2.8e-7.  What bounds the walk is the chain of a chunk (3,100 cycles: the products of S by W
// and of u by k 650 to 730 each, u itself 600, the tensor cores 39 % busy with two warps a scheduler).
//
// ExiledOfCode/KuiperLLama has no recurrent mixer (its mixer is mha_kernel.cu:61,74-106).
#include "pieces.cuh"

namespace kl {

constexpr int DC = 32;                     // tokens of a chunk
constexpr int DC_COLS = 16;                // columns of S of a CTA of the walk
constexpr int DC_THREADS = 256;            // of the CTAs that do not walk
constexpr int DC_RUN = 8;                  // tokens of a warp that prepares
constexpr int DC_MS = DC + 4;              // row stride of a chunk's products in shared memory
constexpr int DC_FACTORS = 128;            // floats: G_t, A(t, C), whether the chunk goes token by token, padding to 256 bytes' multiple
constexpr float DC_MOST = 1048576.f;       // of q and v; S grows by v's at most
constexpr float DC_MOST_S = DC_MOST * DC_MOST * DC_MOST;

struct DeltaChunkArgs {
    float* prep; float* bg;                // [rows, C] q | k | v, [rows, 2 H] beta | decay
    const float* taps_w; const float* A_log; const float* dt_bias;
    float q_scale, unit_eps;
    float* state; long long ld_state;      // S of a slot, [H, d, dv]
    float* out;                            // [rows, H * dv]
    const int* cu_tokens; const int* seq_slots;
    // what the walk copies as it lies
    unsigned char* qk;                     // [chunks, G]: q, then k, in three pieces [3][DC][NP] each
    unsigned char* wm;                     // [chunks, H]: W in three pieces [3][DC][NP], the weights in three pieces [3][DC][DC], the factors
    float* ub;                             // [chunks, H, dv / 16, DC, 16]: T (beta V)
    int H, G, d, dv;
    int chunk0, span;                      // the chunks of every sequence that this launch works: `span` of them from chunk0 on (0: all)
    // the projections, and the convolution's state behind S, which moves on in the walk (see recurrent.cu)
    const bf16* proj; long long ld; int conv_col, b_col, a_col; long long conv_off;
};
constexpr int DC_TAPS = 4;

template <int NP> constexpr int dc_w_bytes() { return 3 * DC * NP * 2; }
template <int NP> constexpr int dc_wm_bytes() { return dc_w_bytes<NP>() + 3 * DC * DC * 2 + DC_FACTORS * 4; }
// The place of a chunk that starts at row `row0` of sequence s among all chunks: a sequence's chunks follow one another, and no two share one.
__device__ __forceinline__ size_t dc_entry(int row0, int s) { return (size_t)(row0 / DC + s); }
// The same in a portion of `span` chunks a sequence, from chunk0 on: first row of the portion's first chunk, and its place.
__device__ __forceinline__ int dc_first(const DeltaChunkArgs& A, int s) { return A.cu_tokens[s] + A.chunk0 * DC; }
__device__ __forceinline__ size_t dc_entry0(const DeltaChunkArgs& A, int s) { return A.span > 0 ? (size_t)s * A.span : dc_entry(A.cu_tokens[s], s); }
__device__ __forceinline__ bool dc_wild(float x, float most) { return !(fabsf(x) <= most); }

// ------------------------------------------------------------------------------------------ convolution, unit lengths, gates
__device__ __forceinline__ float dc_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
// blockIdx.x * 8 + warp: a run of DC_RUN tokens; blockIdx.z: a key head (q and k), then blocks of 128 channels of v, then the gates.  A lane has four
// neighbouring channels; 128 channels are a head of q or k at most.
__global__ void __launch_bounds__(DC_THREADS)
dc_prepare_kernel(const DeltaChunkArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.y, lane = threadIdx.x & 31, item = blockIdx.z;
    const int first = A.cu_tokens[s], n_new = A.cu_tokens[s + 1] - first, t0 = (blockIdx.x * (DC_THREADS / 32) + (threadIdx.x >> 5)) * DC_RUN;
    if (t0 >= n_new) return;
    const int n = min(DC_RUN, n_new - t0), d = A.d, V = A.H * A.dv, C = 2 * A.G * d + V, v_items = (V + 127) / 128;
    if (item >= A.G + v_items) {                           // beta and the decay of (token, head)
        for (int e = lane; e < n * A.H; e += 32) {
            const int t = e / A.H, h = e - t * A.H;
            const bf16* p = A.proj + (size_t)(first + t0 + t) * A.ld;
            const float z = to_f32(p[A.a_col + h]) + A.dt_bias[h];
            float* o = A.bg + (size_t)(first + t0 + t) * 2 * A.H;
            o[h] = dc_sigmoid(to_f32(p[A.b_col + h]));
            o[A.H + h] = expf(-expf(A.A_log[h]) * (z > 20.f ? z : log1pf(expf(z))));
        }
        return;
    }
    const bool keys = item < A.G;
    const int width = keys ? d : min(128, V - (item - A.G) * 128);
    const bool on = lane * 4 < width;
    const int c[2] = {(keys ? item * d : 2 * A.G * d + (item - A.G) * 128) + (on ? lane * 4 : 0), (A.G + item) * d + (on ? lane * 4 : 0)};        // q (or v), and k
    const float* cs = A.state + (size_t)A.seq_slots[s] * A.ld_state + A.conv_off;
    // four channels of a run's tokens and of the three inputs before it (from the state where the step does not hold them), all on their way together
    constexpr int BEFORE = DC_TAPS - 1;
    uint2 raw[2][DC_RUN];
    float w[2][4][DC_TAPS], x[2][4][BEFORE];               // the taps, and the inputs before a token, oldest first
    auto open = [](const uint2& v, float (&y)[4]) {
        y[0] = __uint_as_float(v.x << 16); y[1] = __uint_as_float(v.x & 0xffff0000u); y[2] = __uint_as_float(v.y << 16); y[3] = __uint_as_float(v.y & 0xffff0000u);
    };
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (i == 1 && !keys) break;
        const bf16* p = A.proj + (size_t)(first + t0) * A.ld + A.conv_col + c[i];
#pragma unroll
        for (int t = 0; t < DC_RUN; ++t) raw[i][t] = t < n ? *reinterpret_cast<const uint2*>(p + (size_t)t * A.ld) : make_uint2(0u, 0u);
#pragma unroll
        for (int j = 0; j < BEFORE; ++j) {
            float y[4];
            if (t0 + j >= BEFORE) {
                open(*reinterpret_cast<const uint2*>(p + (long long)(j - BEFORE) * A.ld), y);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) y[e] = cs[(size_t)(t0 + j) * C + c[i] + e];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) x[i][e][j] = y[e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float4 taps = *reinterpret_cast<const float4*>(A.taps_w + (size_t)(c[i] + e) * DC_TAPS);
            w[i][e][0] = taps.x; w[i][e][1] = taps.y; w[i][e][2] = taps.z; w[i][e][3] = taps.w;
        }
    }
#pragma unroll
    for (int t = 0; t < DC_RUN; ++t) {
        if (t >= n) break;
        float y[2][4], ss[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (i == 1 && !keys) break;
            float now[4];
            open(raw[i][t], now);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < BEFORE; ++j) sum = fmaf(w[i][e][j], x[i][e][j], sum);
                sum = fmaf(w[i][e][BEFORE], now[e], sum);
#pragma unroll
                for (int j = 0; j < BEFORE - 1; ++j) x[i][e][j] = x[i][e][j + 1];
                x[i][e][BEFORE - 1] = now[e];
                y[i][e] = on ? sum * dc_sigmoid(sum) : 0.f;
                ss[i] = fmaf(y[i][e], y[i][e], ss[i]);
            }
        }
        float* o = A.prep + (size_t)(first + t0 + t) * C;
        if (keys) {
            const float fq = A.q_scale / sqrtf(warp_sum(ss[0]) + A.unit_eps), fk = 1.0f / sqrtf(warp_sum(ss[1]) + A.unit_eps);
            if (on) {
                *reinterpret_cast<float4*>(o + c[0]) = make_float4(y[0][0] * fq, y[0][1] * fq, y[0][2] * fq, y[0][3] * fq);
                *reinterpret_cast<float4*>(o + c[1]) = make_float4(y[1][0] * fk, y[1][1] * fk, y[1][2] * fk, y[1][3] * fk);
            }
        } else if (on) {
            *reinterpret_cast<float4*>(o + c[0]) = make_float4(y[0][0], y[0][1], y[0][2], y[0][3]);
        }
    }
}

// ------------------------------------------------------------------------------------------ what does not depend on S
template <int NP>
struct DcHead {                            // shared memory, in bytes: q, later v, in pieces; k in pieces, later W; A, L, the weights, T; T's two forms in pieces
    static constexpr int VP = 128;         // columns of v at a time
    static constexpr int Q_BYTES = 3 * DC * (NP > VP ? NP : VP) * 2;
    static constexpr int K = Q_BYTES, A = K + dc_w_bytes<NP>(), L = A + DC * DC_MS * 4, M = L + DC * DC_MS * 4, T = M + DC * DC_MS * 4, TP = T + DC * DC_MS * 4,
                         SC = TP + 2 * 3 * DC * DC * 2, BYTES = SC + 4 * DC * 4;
};
// D[32 tokens, 16 columns a warp] = T (three pieces) times rows of tokens (three pieces, W columns a row), columns from col0 on
template <int W>
__device__ __forceinline__ void dc_times(const bf16* T, const bf16* rows, int col0, int lane, float (&d)[2][2][4]) {
    float small[2][2][4];
    uint32_t f[2][3][2][2];
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            uint32_t w[4];
            pc_ldm4t(smem_u32(rows + x * DC * W + pc_at<W>(ks * 16 + (lane & 15), col0 / 8 + (lane >> 4))), w);
            f[ks][x][0][0] = w[0]; f[ks][x][0][1] = w[1]; f[ks][x][1][0] = w[2]; f[ks][x][1][1] = w[3];
        }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int ks = 0; ks <= mt; ++ks) {                 // (T is zero above the diagonal)
            uint32_t a[3][4];
#pragma unroll
            for (int x = 0; x < 3; ++x) pc_ldm4(smem_u32(T + x * DC * DC + pc_at<DC>(mt * 16 + (lane & 15), ks * 2 + (lane >> 4))), a[x]);
            if (ks == 0) {
                pc_mma33<2, true>(d[mt], small[mt], a, f[0]);
            } else {
                float more[2][4];
                pc_mma33<2, false>(more, small[mt], a, f[1]);
                pc_add<2>(d[mt], more);
            }
        }
    pc_add<2>(d[0], small[0]);
    pc_add<2>(d[1], small[1]);
}
template <int NP>
__global__ void __launch_bounds__(DC_THREADS, 2)
dc_head_kernel(const DeltaChunkArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    typedef DcHead<NP> H;
    extern __shared__ __align__(256) unsigned char dc_raw[];
    bf16 *Qs = reinterpret_cast<bf16*>(dc_raw), *Ks = reinterpret_cast<bf16*>(dc_raw + H::K), *Tp = reinterpret_cast<bf16*>(dc_raw + H::TP);
    float *As = reinterpret_cast<float*>(dc_raw + H::A), *Ls = reinterpret_cast<float*>(dc_raw + H::L), *Ms = reinterpret_cast<float*>(dc_raw + H::M),
          *Ts = reinterpret_cast<float*>(dc_raw + H::T), *sc = reinterpret_cast<float*>(dc_raw + H::SC);
    float *beta = sc, *from = sc + DC, *to = sc + 2 * DC, *bfrom = sc + 3 * DC;            // beta_t, G_t, A(t, C), beta_t G_t
    const int s = blockIdx.z, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = dc_first(A, s) + blockIdx.x * DC, live = min(DC, A.cu_tokens[s + 1] - row0);
    if (live <= 0) return;
    const size_t entry = dc_entry0(A, s) + blockIdx.x;
    const int d = A.d, dv = A.dv, share = A.H / A.G, g = h / share, C = 2 * A.G * d + A.H * dv;
    unsigned char* wm = A.wm + (entry * A.H + h) * dc_wm_bytes<NP>();
    unsigned char* qk = h % share == 0 ? A.qk + (entry * A.G + g) * 2 * dc_w_bytes<NP>() : nullptr;
    bool wild = false;
    // rows of floats in pieces into a tile of rows of W elements (and, as they lie there, to `out`)
    auto pieces = [&](const float4& x0, const float4& x1, bf16* tile, int at, int plane, bf16* out) {
        uint32_t w[3][4];
        pc_split(x0.x, x0.y, w[0][0], w[1][0], w[2][0]);
        pc_split(x0.z, x0.w, w[0][1], w[1][1], w[2][1]);
        pc_split(x1.x, x1.y, w[0][2], w[1][2], w[2][2]);
        pc_split(x1.z, x1.w, w[0][3], w[1][3], w[2][3]);
#pragma unroll
        for (int y = 0; y < 3; ++y) {
            const uint4 v = make_uint4(w[y][0], w[y][1], w[y][2], w[y][3]);
            *reinterpret_cast<uint4*>(tile + y * plane + at) = v;
            if (out != nullptr) *reinterpret_cast<uint4*>(out + y * plane + at) = v;
        }
    };
    auto out_of = [&](const float4& x, float most) { return dc_wild(x.x, most) || dc_wild(x.y, most) || dc_wild(x.z, most) || dc_wild(x.w, most); };
    constexpr int TURNS = DC * NP / 8 / DC_THREADS;
    {
        float4 x[2][TURNS][2];
#pragma unroll
        for (int which = 0; which < 2; ++which)
#pragma unroll
            for (int i = 0; i < TURNS; ++i) {
                const int e = threadIdx.x + DC_THREADS * i, r = e / (NP / 8), p = e % (NP / 8);
                const float* src = A.prep + (size_t)(row0 + r) * C + (size_t)(which ? A.G + g : g) * d + p * 8;
                const bool in = r < live && p * 8 < d;     // d is a multiple of eight
                x[which][i][0] = in ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[which][i][1] = in ? *reinterpret_cast<const float4*>(src + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        if (warp == 0) {                                   // the decays' products, a token a lane
            const float* p = A.bg + (size_t)(row0 + min(lane, live - 1)) * 2 * A.H;
            const float b = lane < live ? p[h] : 0.f, a = lane < live ? p[A.H + h] : 1.f;
            wild = wild || !(b >= 0.f && b <= 1.f) || !(a >= 0.f && a <= 1.f);
            double r = 1.0;                                // (in 64 bits: a product of 32 decays is rounded once)
#pragma unroll
            for (int j = DC - 1; j >= 0; --j) {            // A(j, lane)
                const float aj = __shfl_sync(0xffffffffu, a, j);
                As[lane * DC_MS + j] = j <= lane ? (float)r : 0.f;
                r = j <= lane ? r * aj : 1.0;
            }
            __syncwarp();
            beta[lane] = b;
            from[lane] = lane < live ? (float)r : 0.f;
            bfrom[lane] = (float)(b * r);
            to[lane] = lane < live ? As[(live - 1) * DC_MS + lane] : 0.f;
        }
#pragma unroll
        for (int which = 0; which < 2; ++which)
#pragma unroll
            for (int i = 0; i < TURNS; ++i) {
                const int e = threadIdx.x + DC_THREADS * i, r = e / (NP / 8), p = e % (NP / 8);
                const float most = which ? 1.01f : DC_MOST;                    // (keys are of unit length)
                wild = wild || out_of(x[which][i][0], most) || out_of(x[which][i][1], most);
                pieces(x[which][i][0], x[which][i][1], which ? Ks : Qs, pc_at<NP>(r, p), DC * NP,
                       qk != nullptr ? reinterpret_cast<bf16*>(qk + which * dc_w_bytes<NP>()) : nullptr);
            }
    }
    int any = __syncthreads_or(wild);
    // k . k and q . k, 16 tokens by 16 a warp
    {
        const int rt = warp & 1, ct = (warp >> 1) & 1, which = warp >> 2;
        float sum[2][4], small[2][4];
        pc_zero<2>(sum);
        pc_zero<2>(small);
        if (ct <= rt) {
            const bf16* a_tile = which ? Qs : Ks;
#pragma unroll 2
            for (int ks = 0; ks < NP / 16; ++ks) {
                uint32_t a[3][4], b[3][2][2];
                float more[2][4];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    pc_ldm4(smem_u32(a_tile + i * DC * NP + pc_at<NP>(rt * 16 + (lane & 15), ks * 2 + (lane >> 4))), a[i]);
                    pc_rows<NP, 2>(Ks + i * DC * NP, ct * 16, ks * 2, lane, b[i]);
                }
                pc_mma33<2, false>(more, small, a, b);
                pc_add<2>(sum, more);
            }
            pc_add<2>(sum, small);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = rt * 16 + (lane >> 2) + 8 * (e >> 1), j = ct * 16 + n * 8 + 2 * (lane & 3) + (e & 1);
                const float w = As[t * DC_MS + j] * sum[n][e];
                if (which) Ms[t * DC_MS + j] = w;          // (zero above the diagonal: A is)
                else Ls[t * DC_MS + j] = j < t ? beta[t] * w : 0.f;
            }
    }
    // the first columns of v on their way
    constexpr int V_TURNS = DC * H::VP / 8 / DC_THREADS;
    float4 v[V_TURNS][2];
    auto load_v = [&](int col0) {
#pragma unroll
        for (int i = 0; i < V_TURNS; ++i) {
            const int e = threadIdx.x + DC_THREADS * i, r = e / (H::VP / 8), p = e % (H::VP / 8);
            const float* src = A.prep + (size_t)(row0 + r) * C + 2 * A.G * d + (size_t)h * dv + col0 + p * 8;
            const bool in = r < live && col0 + p * 8 < dv;                     // dv is a multiple of 16
            v[i][0] = in ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][1] = in ? *reinterpret_cast<const float4*>(src + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    load_v(0);
    __syncthreads();
    // T by forward substitution, a column a lane (warp 0); the weights in three pieces (warps 4 to 7)
    if (warp >= 4) {
        const int i = (threadIdx.x - 128) >> 2, q4 = threadIdx.x & 3;
        const float* m = Ms + i * DC_MS + q4 * 8;
        bf16* to_m = reinterpret_cast<bf16*>(wm + dc_w_bytes<NP>());
        uint32_t w[3][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) pc_split(m[2 * u], m[2 * u + 1], w[0][u], w[1][u], w[2][u]);
#pragma unroll
        for (int x = 0; x < 3; ++x) *reinterpret_cast<uint4*>(to_m + x * DC * DC + pc_at<DC>(i, q4)) = make_uint4(w[x][0], w[x][1], w[x][2], w[x][3]);
    } else if (warp == 0) {
        float T[DC];
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            float part[4] = {t == lane ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int q = 0; q < t; q += 4) {
                const float4 l = *reinterpret_cast<const float4*>(Ls + t * DC_MS + q);
                part[0] = fmaf(-l.x, T[q], part[0]);
                if (q + 1 < t) part[1] = fmaf(-l.y, T[q + 1], part[1]);
                if (q + 2 < t) part[2] = fmaf(-l.z, T[q + 2], part[2]);
                if (q + 3 < t) part[3] = fmaf(-l.w, T[q + 3], part[3]);
            }
            T[t] = (part[0] + part[1]) + (part[2] + part[3]);
            Ts[t * DC_MS + lane] = T[t];
        }
    } else if (warp == 1) {
        float* f = reinterpret_cast<float*>(wm + dc_w_bytes<NP>() + 3 * DC * DC * 2);
        f[lane] = from[lane];
        f[DC + lane] = to[lane];
    }
    __syncthreads();
    // T beta and T beta G in three pieces, eight of a row a thread; v over the q that is done with
    {
        const int which = threadIdx.x >> 7, i = (threadIdx.x & 127) >> 2, q4 = threadIdx.x & 3;
        const float *t = Ts + i * DC_MS + q4 * 8, *f = (which ? bfrom : beta) + q4 * 8;
        const float4 x0 = make_float4(t[0] * f[0], t[1] * f[1], t[2] * f[2], t[3] * f[3]), x1 = make_float4(t[4] * f[4], t[5] * f[5], t[6] * f[6], t[7] * f[7]);
        pieces(x0, x1, Tp + which * 3 * DC * DC, pc_at<DC>(i, q4), DC * DC, nullptr);
    }
    const int r = lane >> 2, kc = 2 * (lane & 3);
    for (int col0 = 0; col0 < dv; col0 += H::VP) {
        bool far = false;
#pragma unroll
        for (int i = 0; i < V_TURNS; ++i) {
            const int e = threadIdx.x + DC_THREADS * i;
            far = far || out_of(v[i][0], DC_MOST) || out_of(v[i][1], DC_MOST);
            pieces(v[i][0], v[i][1], Qs, pc_at<H::VP>(e / (H::VP / 8), e % (H::VP / 8)), DC * H::VP, nullptr);
        }
        any |= __syncthreads_or(far);
        if (col0 + H::VP < dv) load_v(col0 + H::VP);
        const int c = col0 + warp * 16;
        if (c < dv) {
            float y[2][2][4];
            dc_times<H::VP>(Tp, Qs, warp * 16, lane, y);
            float* o = A.ub + ((entry * A.H + h) * (dv / DC_COLS) + c / DC_COLS) * DC * DC_COLS;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        *reinterpret_cast<float2*>(o + (mt * 16 + r + 8 * i) * DC_COLS + n * 8 + kc) = make_float2(y[mt][n][2 * i], y[mt][n][2 * i + 1]);
        }
        __syncthreads();
    }
    // W, over k
    {
        float y[2][2][4];
        const bool mine = warp * 16 < NP;
        if (mine) dc_times<NP>(Tp + 3 * DC * DC, Ks, warp * 16, lane, y);
        __syncthreads();
        if (mine) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint32_t w[3];
                        pc_split(y[mt][n][2 * i], y[mt][n][2 * i + 1], w[0], w[1], w[2]);
                        const int at = pc_at<NP>(mt * 16 + r + 8 * i, warp * 2 + n) + kc;
#pragma unroll
                        for (int x = 0; x < 3; ++x) *reinterpret_cast<uint32_t*>(Ks + x * DC * NP + at) = w[x];
                    }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < dc_w_bytes<NP>() / 16; e += DC_THREADS) reinterpret_cast<uint4*>(wm)[e] = reinterpret_cast<const uint4*>(Ks)[e];
    }
    if (threadIdx.x == 0) reinterpret_cast<int*>(wm + dc_w_bytes<NP>() + 3 * DC * DC * 2)[2 * DC] = any;
}

// ------------------------------------------------------------------------------------------ the walk over the chunks
// Shared memory, in bytes: two of q and k, of W, the weights and the factors, and of T (beta V); then the warps' shares of S^T W and of S^T q, U in
// three pieces (as it is and with the decays to the chunk's end), two barriers.
template <int NP>
struct DcWalk {
    static constexpr int WARPS = NP / 16, QK_BYTES = 2 * dc_w_bytes<NP>(), WM_BYTES = dc_wm_bytes<NP>(), UB_BYTES = DC * DC_COLS * 4;
    static constexpr int WM = 2 * QK_BYTES, UB = WM + 2 * WM_BYTES, SHARE = UB + 2 * UB_BYTES, U = SHARE + WARPS * 8 * 512, BARS = U + 2 * 2 * 3 * 512, BYTES = BARS + 16;
    static_assert(QK_BYTES % 256 == 0 && WM_BYTES % 256 == 0 && BYTES <= 227 * 1024, "dc_walk_kernel: shared memory");
    static_assert(WARPS * 4 * 512 >= NP * DC_COLS * 4, "what dc_tokens borrows");
};

// A chunk's tokens one by one, S [NP][DC_COLS] in shared memory; part: a float a thread
template <int NP>
__device__ __noinline__ void dc_tokens(const DeltaChunkArgs& A, float* S, float* part, int row0, int live, int h, int g) {
    constexpr int PARTS = NP / 16 * 32 / DC_COLS, ROWS = NP / PARTS;
    const int p = threadIdx.x % DC_COLS, mine = threadIdx.x / DC_COLS, col = blockIdx.x * DC_COLS + p, d = A.d;
    const int C = 2 * A.G * d + A.H * A.dv;
    for (int t = 0; t < live; ++t) {
        const float *x = A.prep + (size_t)(row0 + t) * C, *q = x + (size_t)g * d, *k = x + (size_t)(A.G + g) * d, *b = A.bg + (size_t)(row0 + t) * 2 * A.H;
        const float decay = b[A.H + h];
        auto over = [&](const float* row) {                // the column's S . row, in all threads of the column's first
            float sum = 0.f;
            for (int n = mine * ROWS; n < min(d, (mine + 1) * ROWS); ++n) sum = fmaf(S[n * DC_COLS + p], row[n], sum);
            __syncthreads();
            part[threadIdx.x] = sum;
            __syncthreads();
            sum = part[p];
            for (int i = 1; i < PARTS; ++i) sum += part[p + i * DC_COLS];
            return sum;
        };
        const float u = b[h] * (x[2 * A.G * d + (size_t)h * A.dv + col] - decay * over(k));
        for (int n = mine * ROWS; n < min(d, (mine + 1) * ROWS); ++n) S[n * DC_COLS + p] = fmaf(k[n], u, decay * S[n * DC_COLS + p]);
        const float y = over(q);
        if (mine == 0) A.out[((size_t)(row0 + t) * A.H + h) * A.dv + col] = y;
    }
    __syncthreads();
}

// PART: of a portion of the step's chunks (A.span)
template <int NP, bool PART>
__global__ void __launch_bounds__(NP / 16 * 32, 1)
dc_walk_kernel(const DeltaChunkArgs A) {
    pdl_wait();
    typedef DcWalk<NP> L;
    constexpr int WARPS = L::WARPS, THREADS = WARPS * 32;
    extern __shared__ __align__(256) unsigned char dc_raw[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(dc_raw + L::BARS);
    const int s = blockIdx.z, h = blockIdx.y, d = A.d, dv = A.dv, g = h / (A.H / A.G), C = 2 * A.G * d + A.H * dv;
    const int first = PART ? dc_first(A, s) : A.cu_tokens[s], rest = A.cu_tokens[s + 1] - first, n_new = PART ? min(rest, A.span * DC) : rest;
    if (n_new <= 0) return;
    const int chunks = (n_new + DC - 1) / DC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, kc = 2 * (lane & 3);
    const size_t entry0 = PART ? (size_t)s * A.span : dc_entry(first, s);
    float* slot = A.state + (size_t)A.seq_slots[s] * A.ld_state;
    if (!PART || A.chunk0 == 0) {                          // the convolution's state moves on, a share of the channels a CTA (nothing reads it any more)
        float* cs = slot + A.conv_off;
        const int n_ctas = gridDim.x * gridDim.y, mine = blockIdx.y * gridDim.x + blockIdx.x;
        for (int c = mine * THREADS + threadIdx.x; c < C; c += n_ctas * THREADS)
            for (int m = 0; m < DC_TAPS - 1; ++m) {         // ascending: an old entry is read before it is overwritten
                const int tt = rest - (DC_TAPS - 1) + m;
                cs[(size_t)m * C + c] = tt >= 0 ? to_f32(A.proj[(size_t)(first + tt) * A.ld + A.conv_col + c]) : cs[(size_t)(rest + m) * C + c];
            }
    }
    if (threadIdx.x == 0) {
        mbar_init(bars, 1);
        mbar_init(bars + 1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto copy = [&](int c) {
        if (threadIdx.x == 0 && c < chunks) {
            const int b = c & 1;
            mbar_expect_tx(bars + b, L::QK_BYTES + L::WM_BYTES + L::UB_BYTES);
            pc_bulk(dc_raw + b * L::QK_BYTES, A.qk + ((entry0 + c) * A.G + g) * L::QK_BYTES, L::QK_BYTES, bars + b);
            pc_bulk(dc_raw + L::WM + b * L::WM_BYTES, A.wm + ((entry0 + c) * A.H + h) * L::WM_BYTES, L::WM_BYTES, bars + b);
            pc_bulk(dc_raw + L::UB + b * L::UB_BYTES, A.ub + (((entry0 + c) * A.H + h) * (dv / DC_COLS) + blockIdx.x) * DC * DC_COLS, L::UB_BYTES, bars + b);
        }
    };
    copy(0);
    float S[2][4];                                         // S^T: columns r, r + 8 by rows kc, kc + 1 of two tiles
    float* S_at = slot + ((size_t)h * d + warp * 16 + kc) * dv + blockIdx.x * DC_COLS + r;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[n][e] = warp * 16 + n * 8 + kc + (e & 1) < d ? S_at[(size_t)(n * 8 + (e & 1)) * dv + 8 * (e >> 1)] : 0.f;
    auto large = [&]() {
        unsigned most = 0;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) most = max(most, __float_as_uint(S[n][e]) & 0x7fffffffu);
        return most > __float_as_uint(DC_MOST_S);
    };
    bool wild_state = large();
    float4* shares = reinterpret_cast<float4*>(dc_raw + L::SHARE) + lane;      // [S^T W, S^T q][warp][4 tiles of 8 tokens][32]
    uint4* U = reinterpret_cast<uint4*>(dc_raw + L::U) + lane;                 // [as it is, decayed][step][piece][32]
    const int ut = warp < 4 ? warp : -1, yt = WARPS == 8 ? warp - 4 : warp;    // the tiles of tokens whose u and y the warp makes
    const uint32_t row_lane = ((lane & 7) + ((lane >> 4) << 3)) * NP * 2 + ((((lane >> 3) & 1) ^ (lane & 7)) << 4);
    const uint32_t k_lane = (lane & 15) * NP * 2 + (((lane >> 4) ^ (lane & 7)) << 4);
    const uint32_t base = smem_u32(dc_raw);

    auto sum_of = [&](int which, int tile) {
        const float4* share = shares + (which * WARPS * 4 + tile) * 32;
        float4 y = share[0];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) {
            const float4 more = share[w * 4 * 32];
            y.x += more.x; y.y += more.y; y.z += more.z; y.w += more.w;
        }
        return y;
    };
    // S^T of the warp's 16 rows (in pieces) by W or q, all 32 tokens: the warp's share
    auto product = [&](int which, uint32_t at, const uint32_t (&a)[3][4]) {
        uint32_t f[3][4][2];
        float Y[4][4], small[4][4];
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int n = 0; n < 4; n += 2) {
                uint32_t w[4];
                pc_ldm4(at + (x * DC + n * 8) * NP * 2, w);
                f[x][n][0] = w[0]; f[x][n][1] = w[1]; f[x][n + 1][0] = w[2]; f[x][n + 1][1] = w[3];
            }
        pc_mma33<4, true>(Y, small, a, f);
#pragma unroll
        for (int n = 0; n < 4; ++n)
            shares[((which * WARPS + warp) * 4 + n) * 32] = make_float4(Y[n][0] + small[n][0], Y[n][1] + small[n][1], Y[n][2] + small[n][2], Y[n][3] + small[n][3]);
    };
    // the y of 8 tokens of chunk c, whose shares of S^T q are whole: `own` is what the chunk's own tokens give, `from` G_t
    float own[4] = {0.f, 0.f, 0.f, 0.f}, from[2] = {0.f, 0.f};
    auto finish = [&](int c) {
        const float4 far = sum_of(1, yt);
        float* y = A.out + ((size_t)(first + c * DC + yt * 8 + kc) * A.H + h) * dv + blockIdx.x * DC_COLS + r;
        const int left = n_new - c * DC - yt * 8 - kc;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float f = e == 0 ? far.x : e == 1 ? far.y : e == 2 ? far.z : far.w;
            if ((e & 1) < left) y[(size_t)(e & 1) * A.H * dv + 8 * (e >> 1)] = fmaf(f, from[e & 1], own[e]);
        }
    };
    bool left = false;                                     // the y of the chunk before is to be finished

    for (int c = 0; c < chunks; ++c) {
        const int b = c & 1, row0 = first + c * DC, live = min(DC, n_new - c * DC);
        const unsigned char* wm = dc_raw + L::WM + b * L::WM_BYTES;
        const float* factors = reinterpret_cast<const float*>(wm + dc_w_bytes<NP>() + 3 * DC * DC * 2);
        bool here = false;                                 // (a copy of this CTA's own always arrives; no wait is without a limit)
        for (uint32_t i = 0; i < SPIN_LIMIT && !here; ++i) here = mbar_try_wait(bars + b, (c >> 1) & 1);
        const bool wild = !here || wild_state || reinterpret_cast<const int*>(factors)[2 * DC] != 0;
        const int slow = __syncthreads_or(wild);           // everyone is done with the other buffers and U; the shares of S^T q are whole
        copy(c + 1);
        if (slow) {
            if (left && yt >= 0) finish(c - 1);
            left = false;
            float* St = reinterpret_cast<float*>(dc_raw + L::SHARE);           // [NP][DC_COLS]
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) St[(warp * 16 + n * 8 + kc + (e & 1)) * DC_COLS + r + 8 * (e >> 1)] = S[n][e];
            __syncthreads();
            dc_tokens<NP>(A, St, reinterpret_cast<float*>(dc_raw + L::U), row0, live, h, g);
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] = St[(warp * 16 + n * 8 + kc + (e & 1)) * DC_COLS + r + 8 * (e >> 1)];
            wild_state = large();
            continue;
        }
        uint32_t a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) pc_split(S[e >> 1][2 * (e & 1)], S[e >> 1][2 * (e & 1) + 1], a[0][e], a[1][e], a[2][e]);
        product(0, (base + L::WM + b * L::WM_BYTES + row_lane) ^ (warp << 5), a);
        if (left && yt >= 0) finish(c - 1);
        left = true;
        __syncthreads();                                   // the shares of S^T W
        const uint32_t q_at = (base + b * L::QK_BYTES + row_lane) ^ (warp << 5);
        if (ut >= 0) {                                     // u of 8 tokens, in pieces
            const float4 w = sum_of(0, ut);
            const float* ub = reinterpret_cast<const float*>(dc_raw + L::UB + b * L::UB_BYTES) + (ut * 8 + kc) * DC_COLS + r;
            const float to0 = factors[DC + ut * 8 + kc], to1 = factors[DC + ut * 8 + kc + 1];
            uint32_t* mine = reinterpret_cast<uint32_t*>(U + (ut >> 1) * 3 * 32) + 2 * (ut & 1);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float u0 = ub[8 * e] - (e ? w.z : w.x), u1 = ub[DC_COLS + 8 * e] - (e ? w.w : w.y);
                uint32_t p[3], q[3];
                pc_split(u0, u1, p[0], p[1], p[2]);
                pc_split(u0 * to0, u1 * to1, q[0], q[1], q[2]);
#pragma unroll
                for (int y = 0; y < 3; ++y) { mine[y * 128 + e] = p[y]; mine[768 + y * 128 + e] = q[y]; }
            }
        } else {
            product(1, q_at, a);                           // (the others after the next barrier)
        }
        __syncthreads();                                   // U
        // S^T = its decay + U^T (decayed) k
        {
            const uint32_t at = (base + b * L::QK_BYTES + dc_w_bytes<NP>() + k_lane) ^ (warp << 5);
            float main[2][4], small[2][4], more[2][4];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                uint32_t u[3][4], f[3][2][2];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    uint32_t w[4];
                    pc_ldm4t(at + (x * DC + ks * 16) * NP * 2, w);
                    f[x][0][0] = w[0]; f[x][0][1] = w[1]; f[x][1][0] = w[2]; f[x][1][1] = w[3];
                    const uint4 v = U[(6 + ks * 3 + x) * 32];
                    u[x][0] = v.x; u[x][1] = v.y; u[x][2] = v.z; u[x][3] = v.w;
                }
                if (ks == 0) pc_mma33<2, true>(main, small, u, f); else pc_mma33<2, false>(more, small, u, f);
            }
            const float alpha = factors[live - 1];
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] = fmaf(alpha, S[n][e], (main[n][e] + more[n][e]) + small[n][e]);
        }
        if (ut >= 0) product(1, q_at, a);
        if (yt >= 0) {                                     // what the chunk's own tokens give 8 of them
            const uint32_t at = base + L::WM + b * L::WM_BYTES + dc_w_bytes<NP>() + pc_at<DC>(yt * 8 + (lane & 7), lane >> 3) * 2;
            uint32_t m[3][4];
#pragma unroll
            for (int x = 0; x < 3; ++x) pc_ldm4(at + x * DC * DC * 2, m[x]);
            float first_16[4], lo[4], hi[4] = {0.f, 0.f, 0.f, 0.f}, more[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                if (ks == 0 || yt >= 2) {
                    uint32_t u[3][4];
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        const uint4 v = U[(ks * 3 + x) * 32];
                        u[x][0] = v.x; u[x][1] = v.y; u[x][2] = v.z; u[x][3] = v.w;
                    }
                    if (ks == 0) pc_mma0(lo, u[2], m[0][0], m[0][1]); else pc_mma(lo, u[2], m[0][2], m[0][3]);
                    pc_mma(hi, u[1], m[0][2 * ks], m[0][2 * ks + 1]);
                    pc_mma0(ks ? more : first_16, u[0], m[0][2 * ks], m[0][2 * ks + 1]);
                    pc_mma(lo, u[1], m[1][2 * ks], m[1][2 * ks + 1]);
                    pc_mma(hi, u[0], m[1][2 * ks], m[1][2 * ks + 1]);
                    pc_mma(lo, u[0], m[2][2 * ks], m[2][2 * ks + 1]);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) own[e] = (first_16[e] + more[e]) + (lo[e] + hi[e]);
            from[0] = factors[yt * 8 + kc];
            from[1] = factors[yt * 8 + kc + 1];
        }
    }
    __syncthreads();
    if (left && yt >= 0) finish(chunks - 1);
    pdl_launch_dependents();
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (warp * 16 + n * 8 + kc + (e & 1) < d) S_at[(size_t)(n * 8 + (e & 1)) * dv + 8 * (e >> 1)] = S[n][e];
}

template <int NP>
static int launch_delta_chunked(const DeltaChunkArgs& A, int chunks, int n_seqs, cudaStream_t stream) {
    KL_CUDA(cudaFuncSetAttribute(dc_head_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, DcHead<NP>::BYTES));
    launch_kernel(dc_head_kernel<NP>, dim3(chunks, A.H, n_seqs), DC_THREADS, DcHead<NP>::BYTES, stream, A);
    KL_LAUNCH_CHECK();
    const auto walk = A.span > 0 ? dc_walk_kernel<NP, true> : dc_walk_kernel<NP, false>;
    KL_CUDA(cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, DcWalk<NP>::BYTES));
    launch_kernel_after(walk, dim3(A.dv / DC_COLS, A.H, n_seqs), NP / 16 * 32, DcWalk<NP>::BYTES, stream, A);
    KL_LAUNCH_CHECK();
    return KL_OK;
}
static long long dc_round(long long bytes) { return (bytes + 255) / 256 * 256; }
static long long dc_wm(int d) { return d <= 64 ? dc_wm_bytes<64>() : dc_wm_bytes<128>(); }
static long long dc_qk(int d) { return 2 * (d <= 64 ? dc_w_bytes<64>() : dc_w_bytes<128>()); }

// What a step's scratch holds: what is prepared of every row, and all chunks where they take up to `limit` bytes, else as many chunks of every sequence as
// that (one at least), and the step is worked in portions of so many.
struct DcPlan {
    long long entries, bytes;
    int chunks, span;                      // chunks of the longest sequence; of every sequence in a portion (0: all of them at once)
    DcPlan(int rows, int n_seqs, int max_new, int H, int G, int d, int dv, long long limit) {
        chunks = (max_new + DC - 1) / DC;
        const long long one = (long long)G * dc_qk(d) + (long long)H * (dc_wm(d) + (long long)dv * DC * 4), C = 2LL * G * d + (long long)H * dv;
        entries = rows / DC + n_seqs + 1;
        span = 0;
        if (entries * one > limit) {
            const long long most = limit / one / n_seqs;
            span = most < 1 ? 1 : most < chunks ? (int)most : chunks;
            if ((long long)span * n_seqs < entries) entries = (long long)span * n_seqs;
            else span = 0;
        }
        bytes = dc_round(entries * G * dc_qk(d)) + dc_round(entries * H * dc_wm(d)) + dc_round(entries * H * dv * DC * 4) + dc_round(rows * C * 4) + dc_round(2LL * rows * H * 4);
    }
    int portions() const { return span > 0 ? (chunks + span - 1) / span : 1; }
};

}  // namespace kl

using namespace kl;

// 1 where the chunked form runs these sizes: keys a multiple of 8 up to 128, values one of 16, four taps.
KL_API int kl_delta_chunked_fits(int n_seqs, int H, int G, int d, int dv, int taps) {
    if (n_seqs <= 0 || n_seqs > 65535 || H <= 0 || G <= 0 || H % G || H > 65535 || d <= 0 || d > 128 || d % 8 || dv <= 0 || dv % 16 || taps != DC_TAPS) return 0;
    return G + (2LL * G * d + (long long)H * dv + 127) / 128 + 1 <= 65535;
}
// Bytes of scratch that kl_delta_chunked needs, and in how many portions it works a step whose chunks keep to `limit` bytes (two launches each, and one before).
KL_API long long kl_delta_chunked_scratch(int rows, int n_seqs, int max_new, int H, int G, int d, int dv, long long limit) {
    return DcPlan(rows, n_seqs, max_new, H, G, d, dv, limit).bytes;
}
KL_API int kl_delta_chunked_portions(int rows, int n_seqs, int max_new, int H, int G, int d, int dv, long long limit) {
    return DcPlan(rows, n_seqs, max_new, H, G, d, dv, limit).portions();
}

// What kl_gated_delta_rule does, for bfloat16 rows of proj whose q | k | v start on an 8-byte boundary, rows a multiple of four elements apart.
// scratch: kl_delta_chunked_scratch bytes on a 16-byte boundary.
KL_API int kl_delta_chunked(const void* proj, long long ld, int conv_col, int b_col, int a_col, const float* taps_w, int taps, const float* A_log,
                            const float* dt_bias, float* state, long long ld_state, long long conv_off, float* out, void* scratch, long long limit,
                            const int* cu_tokens, const int* seq_slots, int rows, int n_seqs, int max_new, int H, int G, int d, int dv, float q_scale,
                            float unit_eps, cudaStream_t stream) {
    if (rows <= 0 || n_seqs <= 0 || max_new <= 0) return KL_OK;
    if (!kl_delta_chunked_fits(n_seqs, H, G, d, dv, taps)) return KL_ERR_BAD_SIZE;
    if (((uintptr_t)scratch | (uintptr_t)taps_w) % 16 || (uintptr_t)proj % 8 || conv_col % 4 || ld % 4) return KL_ERR_BAD_ALIGN;
    const long long C = 2LL * G * d + (long long)H * dv;
    const DcPlan plan(rows, n_seqs, max_new, H, G, d, dv, limit);
    DeltaChunkArgs A;
    A.taps_w = taps_w; A.A_log = A_log; A.dt_bias = dt_bias; A.q_scale = q_scale; A.unit_eps = unit_eps;
    A.state = state; A.ld_state = ld_state; A.out = out; A.cu_tokens = cu_tokens; A.seq_slots = seq_slots; A.H = H; A.G = G; A.d = d; A.dv = dv;
    A.proj = (const bf16*)proj; A.ld = ld; A.conv_col = conv_col; A.b_col = b_col; A.a_col = a_col; A.conv_off = conv_off;
    A.chunk0 = 0; A.span = plan.span;
    unsigned char* at = (unsigned char*)scratch;
    A.qk = at; at += dc_round(plan.entries * G * dc_qk(d));
    A.wm = at; at += dc_round(plan.entries * H * dc_wm(d));
    A.ub = (float*)at; at += dc_round(plan.entries * H * dv * DC * 4);
    A.prep = (float*)at; at += dc_round(rows * C * 4);
    A.bg = (float*)at;
    const int run = DC_RUN * (DC_THREADS / 32);
    launch_kernel(dc_prepare_kernel, dim3((max_new + run - 1) / run, n_seqs, G + (H * dv + 127) / 128 + 1), DC_THREADS, 0, stream, A);
    KL_LAUNCH_CHECK();
    for (int i = 0; i < plan.portions(); ++i) {            // (S goes from one portion to the next through the slot, as the 32-bit numbers that it is)
        A.chunk0 = i * plan.span;
        const int chunks = plan.span > 0 ? (plan.span < plan.chunks - A.chunk0 ? plan.span : plan.chunks - A.chunk0) : plan.chunks;
        const int rc = d <= 64 ? launch_delta_chunked<64>(A, chunks, n_seqs, stream) : launch_delta_chunked<128>(A, chunks, n_seqs, stream);
        if (rc != KL_OK) return rc;
    }
    return KL_OK;
}
