// The mixed-head attention of attention_mixed.cu for prompts of bfloat16 rows, with its products on the tensor cores:
//
//   s_h(i, j) = scale * q_h(i) . k_kv(h)(j);   s <- cap * tanh(s / cap);   s <- s - r1_h * ln(1 + r2_h * (i - j))
//   p_h(i, .) = softmax over the visible keys;   w_h(i, j) = sum_g talk[h, g] p_g(i, j);   out_h(i) = gate * sum_j w_h(i, j) v(j)
//
// The same two launches as in attention_mixed_tiled.cu (phase 0 every head's maximum and sum, phase 1 the rest), the same walk over
// chunks of 32 keys by absolute position and the same masks.  A CTA holds 8 consecutive tokens of a sequence with all H heads in
// H / 2 warps; a warp has two heads of one key/value head, so a tile of 16 rows of mma.m16n8k16 is 8 tokens of each:
//
//   scores   S = Q K^T: bfloat16 operands as they are (exact products, 32-bit sums); Q stays in registers
//   mix      W = talk P as a product of [H, H] with [H, 256 (token, key) pairs]: a warp takes columns of 8 keys of one token and writes W
//            over the P it has read
//   values   O += W V
//
// talk, p and w are 32-bit numbers.  They enter the products as the sum of three bfloat16 numbers (24 bits of mantissa); of two such
// operands the six products down to 2^-16 of the leading one are added, smallest first, so nothing is rounded to 16 bits.
// What bounds it is the instructions of a score outside the products: 76 of phase 0's with a tanh for every size of x, an exact quotient and a mask
// for every score, 56 without (0.72 of them a cycle and scheduler; phase 1 98, 0.50; one more in each since a score over its cap is rounded once), and the tiles' uneven numbers of chunks, which several CTAs share
// (`splits0` and `splits1`; phase 1's sums then meet in a third launch).  One prompt (32 heads of 64 on 8, window 1,024, 64 kept keys), us: 2,048 tokens 571
// before, 408 now; 1,024 349 and 177; 64 tokens after 1,500 301 in one piece each and 54 in 16.  With 32-bit multiply-adds throughout
// (attention_mixed_tiled.cu) 2,242 for 2,048.
//
// ExiledOfCode/KuiperLLama's attention is mha_kernel.cu:61,74-106 (one sequence, one query, no window, no bias).
#include "common.cuh"
#include "pieces.cuh"
#include "soft_cap.cuh"

namespace kl {

constexpr int MX_TQ = 8, MX_CH = 32;              // tokens of a CTA, keys of a chunk
constexpr int MX_PQ = MX_CH + 8;                  // floats of a token's row of P: rows 8 banks apart, pairs of a fragment on 32 banks
constexpr int MX_PH = MX_TQ * MX_PQ + 4;          // floats of a head's P: heads 4 banks apart
constexpr int MX_BIAS = MX_TQ + MX_CH;            // distances of a chunk (one more than there are)

struct MixedMmaArgs {
    const bf16* q; long long q_stride;
    const bf16* gate; long long gate_stride;
    bf16* out; long long out_stride;
    const bf16* k_cache; const bf16* v_cache;
    const int* block_table; int blocks_per_seq;
    const int* cu_tokens; const int* seq_slots; const int* seq_starts;
    const float* r1; const float* r2; const float* talk;
    float* ml;                                    // [splits, rows, heads, 2]
    float* part;                                  // [splits, rows, heads * dim]: phase 1 in several pieces, or null
    int* counts;                                  // [rows]: into how many pieces phase 1 cut the row's tile
    int rows, n_seqs, splits0, splits1;           // pieces that a tile's chunks are dealt to at most, in phase 0 and in phase 1
    int kv_heads, window, keep_first;
    float scale, softcap, out_scale;
    float scale_cap, scale_cap_rest;              // scale / softcap as the sum of two numbers: a score times it is rounded once
};

inline size_t mx_smem_bytes(int H, int D, int G, int phase) {
    return (size_t)(phase == 1 ? 3 : 2) * G * MX_CH * D * 2 + (size_t)(H / 2) * 2 * MX_BIAS * 4 +
           (phase == 1 ? (size_t)H * MX_PH * 4 + (size_t)3 * H * (H + 8) * 2 : 0);
}

// What a tile of tokens sees.  Its chunks are dealt to as many pieces as it has chunks, `splits` at most: the pieces follow from where a sequence stands
// and not from what the host knew when it launched (or captured) the kernel.
struct MixedTile {
    int i0, nrows, lo, first, kept, visible;      // position of its first token, tokens, first key in the window, its chunk, chunks of kept keys, chunks in all
    __device__ __forceinline__ MixedTile(const MixedMmaArgs& A, int s, int tile) {
        nrows = min(MX_TQ, A.cu_tokens[s + 1] - A.cu_tokens[s] - tile * MX_TQ);
        i0 = A.seq_starts[s] + tile * MX_TQ;
        lo = A.window > 0 ? max(0, i0 - A.window + 1) : 0;
        first = lo / MX_CH;
        kept = A.window > 0 ? min(first, (A.keep_first + MX_CH - 1) / MX_CH) : 0;
        visible = kept + (i0 + nrows - 1) / MX_CH + 1 - first;
    }
    __device__ __forceinline__ int pieces(int splits) const { return min(splits, visible); }
    __device__ __forceinline__ int chunk(int v) const { return v < kept ? v : v - kept + first; }
};

template <int H, int D, int PHASE>
__global__ void __launch_bounds__(H * 16, PHASE == 1 ? 1 : 512 / (H * 16) + 1)
attention_mixed_mma_kernel(const MixedMmaArgs A) {
    constexpr int THREADS = H * 16, WARPS = H / 2, KS = D / 16, NT = MX_CH / 8;
    pdl_wait();
    extern __shared__ __align__(128) unsigned char mx_raw[];
    const int s = blockIdx.y, tile = gridDim.x - 1 - blockIdx.x;           // late tiles see the most keys: they start first
    const MixedTile span(A, s, tile);
    const int nrows = span.nrows, row0 = A.cu_tokens[s] + tile * MX_TQ, piece = blockIdx.z;
    if (nrows <= 0) return;
    const int pieces = span.pieces(PHASE == 0 ? A.splits0 : A.splits1);
    if (piece >= pieces) return;
    const int G = A.kv_heads;
    const int i0 = span.i0, i_last = i0 + nrows - 1;
    const int keep = A.window > 0 ? A.keep_first : 0;
    const int* table = A.block_table + (size_t)A.seq_slots[s] * A.blocks_per_seq;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h0 = 2 * warp, g = h0 / (H / G);
    const int r = lane >> 2, kc = 2 * (lane & 3);                          // the fragment's token, and its first column of eight

    const size_t tile_elems = (size_t)G * MX_CH * D;
    bf16* Ks = reinterpret_cast<bf16*>(mx_raw);                            // [2][G][32][D]
    bf16* Vs = Ks + 2 * tile_elems;                                        // [G][32][D] (phase 1)
    float* bias = reinterpret_cast<float*>(Vs + (PHASE == 1 ? tile_elems : 0)) + warp * 2 * MX_BIAS;
    float* Ps = reinterpret_cast<float*>(Vs + (PHASE == 1 ? tile_elems : 0)) + WARPS * 2 * MX_BIAS;      // [H][MX_PH] (phase 1)
    bf16* Ts = reinterpret_cast<bf16*>(Ps + H * MX_PH);                    // [3][H][H + 8]: talk in three pieces (phase 1)

    auto copy_chunk = [&](bf16* dst, const bf16* cache, int c) {
        const int j0 = c * MX_CH, valid = min(MX_CH, i_last - j0 + 1);
        const bf16* src = cache + ((size_t)table[j0 / PAGE] * G * PAGE + j0 % PAGE) * D;
        for (int idx = threadIdx.x; idx < G * MX_CH * (D / 8); idx += THREADS) {
            const int row = idx / (D / 8), p = idx % (D / 8), kv = row / MX_CH, j = row % MX_CH;
            const bool in = j < valid;                                     // rows past the last key become zero
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + (size_t)kv * MX_CH * D + pc_at<D>(j, p))),
                         "l"(in ? src + ((size_t)kv * PAGE + j) * D + p * 8 : src), "r"(in ? 16 : 0) : "memory");
        }
    };
    auto commit = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };

    // chunks that neither the window nor the kept first keys reach are skipped; this piece has every `pieces`-th of the others
    int v = piece;
    copy_chunk(Ks, A.k_cache, span.chunk(v));
    commit();
    if (PHASE == 1 && A.talk != nullptr)
        for (int idx = threadIdx.x; idx < H * H / 2; idx += THREADS) {
            const int h = idx / (H / 2), e = idx % (H / 2) * 2;
            const float2 t = *reinterpret_cast<const float2*>(A.talk + (size_t)h * H + e);
            uint32_t a, b, l;
            pc_split(t.x, t.y, a, b, l);
            *reinterpret_cast<uint32_t*>(Ts + (size_t)h * (H + 8) + e) = a;
            *reinterpret_cast<uint32_t*>(Ts + (size_t)(H + h) * (H + 8) + e) = b;
            *reinterpret_cast<uint32_t*>(Ts + (size_t)(2 * H + h) * (H + 8) + e) = l;
        }
    uint32_t qf[KS][4];
    {
        const bf16* q = A.q + (size_t)(row0 + min(r, nrows - 1)) * A.q_stride + (size_t)h0 * D + kc;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int e = 0; e < 4; ++e)                                    // rows of both heads, then eight columns further on
                qf[ks][e] = *reinterpret_cast<const uint32_t*>(q + (e & 1) * D + ks * 16 + (e >> 1) * 8);
    }
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};                // of the token for both heads; phase 1: the maximum and the sum's inverse
    if (PHASE == 1) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float* ml = A.ml + ((size_t)(row0 + min(r, nrows - 1)) * H + h0 + e) * 2;
            const int before = span.pieces(A.splits0);
            for (int z = 0; z < before; ++z) m[e] = fmaxf(m[e], ml[(size_t)z * A.rows * H * 2]);
            for (int z = 0; z < before; ++z) {             // (a piece that saw nothing: its maximum is -inf, its sum 0)
                const float2 x = *reinterpret_cast<const float2*>(ml + (size_t)z * A.rows * H * 2);
                if (x.y > 0.f) l[e] += x.y * expf(x.x - m[e]);
                else if (!(x.y == 0.f)) l[e] = x.y;        // NaN stays
            }
            l[e] = l[e] > 0.f ? 1.0f / l[e] : 0.f;
        }
    }
    const float r1[2] = {A.r1 != nullptr ? A.r1[h0] : 0.f, A.r1 != nullptr ? A.r1[h0 + 1] : 0.f};
    const float r2[2] = {A.r1 != nullptr ? A.r2[h0] : 0.f, A.r1 != nullptr ? A.r2[h0 + 1] : 0.f};
    const int i = i0 + r;
    float O[PHASE == 1 ? D / 8 : 1][4];
#pragma unroll
    for (int n = 0; n < (PHASE == 1 ? D / 8 : 1); ++n) O[n][0] = O[n][1] = O[n][2] = O[n][3] = 0.f;

    int buf = 0;
    for (; v < span.visible; v += pieces) {
        const int c = span.chunk(v), j0 = c * MX_CH;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                                   // this chunk's keys are here; the chunk before is done with the buffers
        if (PHASE == 1) copy_chunk(Vs, A.v_cache, c);
        commit();
        if (v + pieces < span.visible) copy_chunk(Ks + (buf ^ 1) * tile_elems, A.k_cache, span.chunk(v + pieces));
        commit();
        // ---- scores: 8 tokens of two heads by 32 keys
        float S[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) S[n][0] = S[n][1] = S[n][2] = S[n][3] = 0.f;
        const bf16* K = Ks + buf * tile_elems + (size_t)g * MX_CH * D;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[4];
                pc_ldm4(smem_u32(K + pc_at<D>(n * 8 + (lane & 7) + ((lane >> 4) << 3), ks * 2 + ((lane >> 3) & 1))), b);
                pc_mma(S[n], qf[ks], b[0], b[1]);
                pc_mma(S[n + 1], qf[ks], b[2], b[3]);
            }
        if (A.r1 != nullptr) {                                             // the bias depends on i - j alone: 39 values for the chunk
            __syncwarp();
            for (int x = lane; x < 2 * MX_BIAS; x += 32) {
                const int e = x / MX_BIAS;
                bias[x] = r1[e] * log1pf(r2[e] * (float)max(0, i0 - j0 - (MX_CH - 1) + x - e * MX_BIAS));
            }
            __syncwarp();
        }
        // (a chunk that every token of a whole tile sees has no masks)
        const bool inside = nrows == MX_TQ && j0 + MX_CH - 1 <= i0 && (A.window == 0 || i_last - j0 < A.window || j0 + MX_CH <= keep);
        auto visible = [&](int n, int e) {
            const int pos = j0 + n * 8 + kc + (e & 1);
            return r < nrows && pos <= i && (A.window == 0 || i - pos < A.window || pos < keep);
        };
        if (A.softcap > 0.f) {
            float most = 0.f;                                              // of the lane's visible scores, all of one token: its result does not depend on what it does not see
            if (inside) {
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) most = fmaxf(most, fabsf(S[n][e]));
            } else {
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) most = visible(n, e) ? fmaxf(most, fabsf(S[n][e])) : most;
            }
            if (most * fabsf(A.scale_cap) > CAP_SMALL) {
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[n][e] = tanhf(cap_quotient(S[n][e], A.scale_cap, A.scale_cap_rest));
            } else {
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[n][e] = cap_tanh(cap_small_quotient(S[n][e], A.scale_cap, A.scale_cap_rest));
            }
        }
        const float factor = A.softcap > 0.f ? A.softcap : A.scale;
        if (A.r1 != nullptr) {
            const float* at = bias + r + (MX_CH - 1) - kc;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] = fmaf(S[n][e], factor, -at[(e >> 1) * MX_BIAS - n * 8 - (e & 1)]);
        } else {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] *= factor;
        }
        if (!inside)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] = visible(n, e) ? S[n][e] : -INFINITY;
        if constexpr (PHASE == 0) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float top = m[e];
#pragma unroll
                for (int n = 0; n < NT; ++n) top = fmaxf(top, fmaxf(S[n][2 * e], S[n][2 * e + 1]));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                if (top == -INFINITY) continue;                            // (the four lanes of a token agree)
                float sum = 0.f;
#pragma unroll
                for (int n = 0; n < NT; ++n) sum += expf(S[n][2 * e] - top) + expf(S[n][2 * e + 1] - top);
                l[e] = l[e] * expf(m[e] - top) + sum;
                m[e] = top;
            }
        } else {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float2 p;
                    p.x = expf(S[n][2 * e] - m[e]) * l[e];                 // exp(-inf) = 0 for a key that is not visible
                    p.y = expf(S[n][2 * e + 1] - m[e]) * l[e];
                    if (r >= nrows) p = make_float2(0.f, 0.f);
                    *reinterpret_cast<float2*>(Ps + (h0 + e) * MX_PH + r * MX_PQ + n * 8 + kc) = p;
                }
            asm volatile("cp.async.wait_group 1;" ::: "memory");           // the values are here (the next keys may still be on their way)
            __syncthreads();                                               // and every head's p of the chunk
            if (A.talk != nullptr) {
                // ---- mix: columns of 8 keys of one token, all heads
#pragma unroll 1
                for (int t = warp; t < MX_TQ * NT; t += WARPS) {
                    float* P = Ps + (t / NT) * MX_PQ + (t % NT) * 8;
                    uint32_t b[3][H / 16][2];
#pragma unroll
                    for (int ks = 0; ks < H / 16; ++ks)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float* p = P + (ks * 16 + kc + 8 * e) * MX_PH + r;
                            pc_split(p[0], p[MX_PH], b[0][ks][e], b[1][ks][e], b[2][ks][e]);
                        }
                    __syncwarp();                                          // all heads' p of these columns are read: w takes their place
#pragma unroll
                    for (int mt = 0; mt < H / 16; ++mt) {
                        float w[4] = {0.f, 0.f, 0.f, 0.f};
                        uint32_t a[3][H / 16][4];
#pragma unroll
                        for (int x = 0; x < 3; ++x)
#pragma unroll
                            for (int ks = 0; ks < H / 16; ++ks)
                                pc_ldm4(smem_u32(Ts + (size_t)(x * H + mt * 16 + (lane & 15)) * (H + 8) + ks * 16 + (lane >> 4) * 8), a[x][ks]);
#pragma unroll
                        for (int ks = 0; ks < H / 16; ++ks) {
                            pc_mma(w, a[2][ks], b[0][ks][0], b[0][ks][1]);
                            pc_mma(w, a[1][ks], b[1][ks][0], b[1][ks][1]);
                            pc_mma(w, a[0][ks], b[2][ks][0], b[2][ks][1]);
                        }
#pragma unroll
                        for (int ks = 0; ks < H / 16; ++ks) {
                            pc_mma(w, a[1][ks], b[0][ks][0], b[0][ks][1]);
                            pc_mma(w, a[0][ks], b[1][ks][0], b[1][ks][1]);
                        }
#pragma unroll
                        for (int ks = 0; ks < H / 16; ++ks) pc_mma(w, a[0][ks], b[0][ks][0], b[0][ks][1]);
                        *reinterpret_cast<float2*>(P + (mt * 16 + r) * MX_PH + kc) = make_float2(w[0], w[1]);
                        *reinterpret_cast<float2*>(P + (mt * 16 + 8 + r) * MX_PH + kc) = make_float2(w[2], w[3]);
                    }
                }
                __syncthreads();
            } else {
                __syncwarp();                                              // a warp reads back what its own lanes wrote
            }
            // ---- O += W V
            const bf16* V = Vs + (size_t)g * MX_CH * D;
#pragma unroll
            for (int ks = 0; ks < MX_CH / 16; ++ks) {
                uint32_t a[3][4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 w = *reinterpret_cast<const float2*>(Ps + (h0 + (e & 1)) * MX_PH + r * MX_PQ + ks * 16 + (e >> 1) * 8 + kc);
                    pc_split(w.x, w.y, a[0][e], a[1][e], a[2][e]);
                }
#pragma unroll
                for (int n = 0; n < D / 8; n += 2) {
                    uint32_t b[4];
                    pc_ldm4t(smem_u32(V + pc_at<D>(ks * 16 + (lane & 15), n + (lane >> 4))), b);
#pragma unroll
                    for (int x = 2; x >= 0; --x) {
                        pc_mma(O[n], a[x], b[0], b[1]);
                        pc_mma(O[n + 1], a[x], b[2], b[3]);
                    }
                }
            }
            __syncwarp();                                                  // the warp's rows of W are read before its next p are written there
        }
        buf ^= 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    pdl_launch_dependents();
    if (r >= nrows) return;
    const size_t row = (size_t)(row0 + r);
    if constexpr (PHASE == 0) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            l[e] += __shfl_xor_sync(0xfu << (lane & ~3), l[e], 1);
            l[e] += __shfl_xor_sync(0xfu << (lane & ~3), l[e], 2);
            if ((lane & 3) == 0) *reinterpret_cast<float2*>(A.ml + (((size_t)piece * A.rows + row) * H + h0 + e) * 2) = make_float2(m[e], l[e]);
        }
    } else if (A.splits1 > 1) {
        if (piece == 0 && warp == 0 && (lane & 3) == 0) A.counts[row] = pieces;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float* o = A.part + ((size_t)piece * A.rows + row) * H * D + (size_t)(h0 + e) * D + kc;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) *reinterpret_cast<float2*>(o + n * 8) = make_float2(O[n][2 * e], O[n][2 * e + 1]);
        }
    } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float f = A.out_scale;
            if (A.gate != nullptr) f *= 1.0f / (1.0f + expf(-to_f32(A.gate[row * A.gate_stride + h0 + e])));
            bf16* o = A.out + row * A.out_stride + (size_t)(h0 + e) * D + kc;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) *reinterpret_cast<__nv_bfloat162*>(o + n * 8) = __floats2bfloat162_rn(O[n][2 * e] * f, O[n][2 * e + 1] * f);
        }
    }
}

// The pieces of phase 1 put together: four neighbouring columns of a row a thread, pieces in ascending order.
__global__ void __launch_bounds__(256)
attention_mixed_mma_reduce_kernel(const MixedMmaArgs A, int heads, int dim) {
    pdl_launch_dependents();
    pdl_wait();
    const int width = heads * dim / 4;
    const int idx = blockIdx.x * 256 + threadIdx.x, row = idx / width, c = (idx - row * width) * 4;
    if (row >= A.cu_tokens[A.n_seqs]) return;                      // (a padding row has no sums)
    const int pieces = A.counts[row];
    const float* p = A.part + (size_t)row * heads * dim + c;
    float4 y = *reinterpret_cast<const float4*>(p);
    for (int z = 1; z < pieces; ++z) {
        const float4 x = *reinterpret_cast<const float4*>(p + (size_t)z * A.rows * heads * dim);
        y.x += x.x; y.y += x.y; y.z += x.z; y.w += x.w;
    }
    float f = A.out_scale;
    if (A.gate != nullptr) f *= 1.0f / (1.0f + expf(-to_f32(A.gate[row * A.gate_stride + c / dim])));
    bf16* o = A.out + row * A.out_stride + c;
    *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(y.x * f, y.y * f);
    *reinterpret_cast<__nv_bfloat162*>(o + 2) = __floats2bfloat162_rn(y.z * f, y.w * f);
}

template <int H, int D, int PHASE>
static int launch_mixed_mma(const MixedMmaArgs& A, dim3 grid, cudaStream_t stream) {
    const size_t smem = mx_smem_bytes(H, D, A.kv_heads, PHASE);
    KL_CUDA(cudaFuncSetAttribute(attention_mixed_mma_kernel<H, D, PHASE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_kernel(attention_mixed_mma_kernel<H, D, PHASE>, dim3(grid.x, grid.y, PHASE == 0 ? A.splits0 : A.splits1), H * 16, smem, stream, A);
    KL_LAUNCH_CHECK();
    return KL_OK;
}

}  // namespace kl

using namespace kl;

// Whether kl_attention_mixed_mma runs these sizes: 16 or 32 heads, an even number of them to a key/value head, keys and values of 32 or
// 64 (larger heads, and 16 key/value heads of 64, leave no room for the chunks beside P), and steps of more than four tokens a sequence (a tile of eight mostly
// empty is no gain).
KL_API int kl_attention_mixed_mma_fits(int heads, int kv_heads, int dim, int vdim, int dtype, int max_new) {
    return dtype == KL_BF16 && (heads == 16 || heads == 32) && kv_heads > 0 && heads % kv_heads == 0 && heads / kv_heads % 2 == 0 && dim == vdim &&
           (dim == 32 || dim == 64) && max_new > 4 && mx_smem_bytes(heads, dim, kv_heads, 1) <= 227 * 1024;
}

// ml: float32 [splits0, rows, heads, 2]; part: float32 [splits1, rows, heads * dim] on a 16-byte boundary, and counts: int32 [rows], where splits1 > 1.  q and out: rows and
// heads on 4-byte boundaries; the caches on 16-byte ones.
KL_API int kl_attention_mixed_mma(const void* q, long long q_stride, const void* gate, long long gate_stride, void* out, long long out_stride,
                                  const void* k_cache, const void* v_cache, const int* block_table, int blocks_per_seq, const int* cu_tokens,
                                  const int* seq_slots, const int* seq_starts, int rows, int n_seqs, int max_new, int heads, int kv_heads,
                                  int dim, float scale, float softcap, const float* r1, const float* r2, const float* talk, int window,
                                  int keep_first, float out_scale, int splits0, int splits1, float* ml, float* part, int* counts, cudaStream_t stream) {
    if (rows <= 0 || n_seqs <= 0 || max_new <= 0) return KL_OK;
    if (!kl_attention_mixed_mma_fits(heads, kv_heads, dim, dim, KL_BF16, max_new) || window < 0 || keep_first < 0 || n_seqs > 65535) return KL_ERR_BAD_SIZE;
    if ((r1 == nullptr) != (r2 == nullptr) || ml == nullptr || splits0 < 1 || splits1 < 1 || splits0 > 64 || splits1 > 64) return KL_ERR_BAD_SIZE;
    if (splits1 > 1 && (part == nullptr || counts == nullptr || (uintptr_t)part % 16)) return KL_ERR_BAD_ALIGN;
    if (((uintptr_t)q | (uintptr_t)out) % 4 || q_stride % 2 || out_stride % 2 || ((uintptr_t)k_cache | (uintptr_t)v_cache) % 16 || (uintptr_t)talk % 8 ||
        (uintptr_t)ml % 8) return KL_ERR_BAD_ALIGN;
    MixedMmaArgs A;
    A.q = (const bf16*)q; A.q_stride = q_stride; A.gate = (const bf16*)gate; A.gate_stride = gate_stride; A.out = (bf16*)out; A.out_stride = out_stride;
    A.k_cache = (const bf16*)k_cache; A.v_cache = (const bf16*)v_cache; A.block_table = block_table; A.blocks_per_seq = blocks_per_seq;
    A.cu_tokens = cu_tokens; A.seq_slots = seq_slots; A.seq_starts = seq_starts; A.r1 = r1; A.r2 = r2; A.talk = talk; A.ml = ml;
    A.kv_heads = kv_heads; A.window = window; A.keep_first = keep_first; A.scale = scale; A.softcap = softcap; A.out_scale = out_scale;
    cap_parts(scale, softcap, A.scale_cap, A.scale_cap_rest);
    A.rows = rows; A.n_seqs = n_seqs; A.splits0 = splits0; A.splits1 = splits1; A.part = part; A.counts = counts;
    const dim3 grid((max_new + MX_TQ - 1) / MX_TQ, n_seqs);
    int err = KL_OK;
#define KL_MX(H_, D_)                                                                       \
    do {                                                                                    \
        err = launch_mixed_mma<H_, D_, 0>(A, grid, stream);                                 \
        if (err == KL_OK) err = launch_mixed_mma<H_, D_, 1>(A, grid, stream);               \
    } while (0)
    if (heads == 32 && dim == 64) KL_MX(32, 64);
    else if (heads == 32) KL_MX(32, 32);
    else if (dim == 64) KL_MX(16, 64);
    else KL_MX(16, 32);
#undef KL_MX
    if (err != KL_OK || splits1 == 1) return err;
    launch_kernel(attention_mixed_mma_reduce_kernel, (int)(((long long)rows * heads * dim / 4 + 255) / 256), 256, 0, stream, A, heads, dim);
    KL_LAUNCH_CHECK();
    return KL_OK;
}
