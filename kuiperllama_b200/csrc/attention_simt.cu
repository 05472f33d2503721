// Causal grouped-query attention over the paged cache, plain SIMT arithmetic in 32 bits.
//
// This is the kernel of the true 32-bit path (prefill and decode) and the fallback of the
// bfloat16 path for sizes and options that the tensor-core kernels refuse (a window, a
// head size that is not on their list; any key size and value sizes up to 512 run here).  One CTA of four warps per
// (token, query head).  Query token t of slot s at position p reads keys lo..p of that
// slot, lo = max(0, p - window + 1) with a window, else 0.  Head h reads kv head
// h / (H / KV); score = (q . k) * scale; softmax with the maximum subtracted; o = sum p v
// (ExiledOfCode/KuiperLLama mha_kernel.cu:61,74-106; there one CTA per head loops over one
// sequence and the scores pass through global memory).
//
// Keys are cut into chunks of 32 by absolute position and the chunks are dealt to the warps
// round-robin, so the order of every sum depends only on the token's own position: the
// result does not change with the way tokens are cut into steps or batched.
//
// attention_simt_kernel reads keys and values where they lie and hides the latency with many CTAs an SM and with loads in batches: 128
// bytes of a key's row, then the values of eight keys, are on their way together (one load at a time made a chunk wait for every 16
// bytes: one token of 300 keys, 32 heads of 64 on 8, 27.3 us, now 10.7; 64 such tokens 116, now 57).
//
// attention_simt_tile_kernel does the same for float32 rows without a window, chunks or distance bias (key and value sizes up to 128):
// a warp copies its chunk of keys and values to shared memory first, as whole lines, and a CTA takes eight neighbouring rows of a
// prompt, which share the copies (TQ = 8), or one row (TQ = 1).  Every token's sums are the same operations in the same order as in the
// kernel above, so its result has the same bits.  Its shared memory leaves one to five CTAs an SM, so it runs only where that is
// no loss (simt_rows_of_a_tile).  One prompt of 777 tokens, 32 heads of 64 on 8: 480 us, 757 with a CTA per token.
//
// Options beyond KuiperLLama's attention: values of another size than the keys (`vd` columns of rows
// that are `v_ld` apart; with v_cache == k_cache and v_ld == hd the values are the leading columns of
// the keys, which is what attention over a shared latent reads), and a sink: a learned number per
// head that joins the softmax's denominator as exp(sink) and has no value; chunks: a token reads the keys of its own chunk
// of `chunk` positions, counted from position 0; and a learned bias by distance: rel[h, min(pos - key, rel_n - 1)] is
// added to the scaled score.
#include "common.cuh"

namespace kl {

constexpr int ATT_WARPS = 4;
constexpr int ATT_MAX_VALUE_DIM = 512;   // value columns per head (32 lanes x PL, PL = 8 or 16)

template <typename T>
__device__ __forceinline__ float dot_row(const T* __restrict__ k, const float* __restrict__ q, int hd);

// four products, added in one order wherever it is used
__device__ __forceinline__ float dot4(const float4 k, const float4 q) {
    return fmaf(k.w, q.w, fmaf(k.z, q.z, fmaf(k.y, q.y, k.x * q.x)));
}

// Head sizes whose rows do not start on 16-byte boundaries take the element-by-element form.
template <typename T>
__device__ __forceinline__ float dot_row_scalar(const T* __restrict__ k, const float* __restrict__ q, int hd) {
    float s = 0.f;
    for (int i = 0; i < hd; ++i) s += to_f32(k[i]) * q[i];
    return s;
}

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ k, const float* __restrict__ q, int hd) {
    if (hd & 3) return dot_row_scalar(k, q, hd);
    float s = 0.f;
    int i = 0;
    for (; i + 32 <= hd; i += 32) {                                  // 128 bytes of the row on their way at a time
        float4 kv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) kv[u] = *reinterpret_cast<const float4*>(k + i + 4 * u);
#pragma unroll
        for (int u = 0; u < 8; ++u) s += dot4(kv[u], *reinterpret_cast<const float4*>(q + i + 4 * u));
    }
    for (; i < hd; i += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(k + i);
        s += dot4(kv, *reinterpret_cast<const float4*>(q + i));
    }
    return s;
}
template <>
__device__ __forceinline__ float dot_row<bf16>(const bf16* __restrict__ k, const float* __restrict__ q, int hd) {
    if (hd & 7) return dot_row_scalar(k, q, hd);
    float s = 0.f;
    for (int i = 0; i < hd; i += 8) {
        const uint4 raw = *reinterpret_cast<const uint4*>(k + i);
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(p[j]);
            s += f.x * q[i + 2 * j] + f.y * q[i + 2 * j + 1];
        }
    }
    return s;
}

template <typename T, int PL>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                      const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                      const int* __restrict__ block_table, int blocks_per_seq,
                      const int* __restrict__ positions, const int* __restrict__ token_slot,
                      int H, int KV, int hd, float scale, int window, int vd, int v_ld, const float* __restrict__ sink, int chunk,
                      const float* __restrict__ rel, int rel_n) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;                               // [hd]
    float* m_s = q_s + hd;                           // [ATT_WARPS]
    float* l_s = m_s + ATT_WARPS;                    // [ATT_WARPS]
    float* acc_s = l_s + ATT_WARPS;                  // [ATT_WARPS][vd]

    const int t = blockIdx.x, h = blockIdx.y;
    const int slot = token_slot[t];
    if (slot < 0) return;                            // a padding row: nothing is written
    const int pos = positions[t];
    const int g = h / (H / KV);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    const T* qrow = q + (size_t)t * q_stride + (size_t)h * hd;
    for (int i = threadIdx.x; i < hd; i += blockDim.x) q_s[i] = to_f32(qrow[i]);
    __syncthreads();

    int lo = window > 0 ? max(0, pos - window + 1) : 0;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    float m = -INFINITY, l = 0.f;
    float acc[PL];
#pragma unroll
    for (int i = 0; i < PL; ++i) acc[i] = 0.f;

    const int* table = block_table + (size_t)slot * blocks_per_seq;
    for (int c = lo / 32 + warp; c * 32 <= pos; c += ATT_WARPS) {
        const int base = c * 32;                                     // 32 keys inside one page
        const int page = table[base / PAGE];
        const size_t page_off = (((size_t)page * KV + g) * PAGE + (base % PAGE)) * (size_t)hd;
        const int key = base + lane;
        const bool valid = key >= lo && key <= pos;
        float s = -INFINITY;
        if (valid) {
            s = dot_row<T>(k_cache + page_off + (size_t)lane * hd, q_s, hd) * scale;
            if (rel != nullptr) s += rel[(size_t)h * rel_n + min(pos - key, rel_n - 1)];
        }
        const float m_new = fmaxf(m, warp_max(s));                   // finite: the chunk holds a valid key
        const float corr = expf(m - m_new);                          // exp(-inf) = 0 at the first chunk
        const float p = valid ? expf(s - m_new) : 0.f;
        l = fmaf(l, corr, warp_sum(p));
        m = m_new;
#pragma unroll
        for (int i = 0; i < PL; ++i) acc[i] *= corr;
        const int j_lo = max(lo - base, 0), j_hi = min(pos - base, 31);
        const T* vbase = v_cache + (((size_t)page * KV + g) * PAGE + (base % PAGE)) * (size_t)v_ld;
        constexpr int U = PL <= 4 ? 8 : 32 / PL;                     // keys whose values are requested together
        int j = j_lo;
        for (; j + U - 1 <= j_hi; j += U) {
            float v[U][PL];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < PL; ++i) v[u][i] = lane + 32 * i < vd ? to_f32(vbase[(size_t)(j + u) * v_ld + lane + 32 * i]) : 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float pj = __shfl_sync(0xffffffffu, p, j + u);
#pragma unroll
                for (int i = 0; i < PL; ++i) acc[i] = fmaf(pj, v[u][i], acc[i]);
            }
        }
        for (; j <= j_hi; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const T* vrow = vbase + (size_t)j * v_ld;
#pragma unroll
            for (int i = 0; i < PL; ++i) {
                const int d = lane + 32 * i;
                if (d < vd) acc[i] = fmaf(pj, to_f32(vrow[d]), acc[i]);
            }
        }
    }
    if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
#pragma unroll
    for (int i = 0; i < PL; ++i) {
        const int d = lane + 32 * i;
        if (d < vd) acc_s[warp * vd + d] = acc[i];
    }
    __syncthreads();
    float M = m_s[0];
#pragma unroll
    for (int w = 1; w < ATT_WARPS; ++w) M = fmaxf(M, m_s[w]);
    const float snk = sink ? sink[h] : -INFINITY;
    M = fmaxf(M, snk);
    float L = sink ? expf(snk - M) : 0.f;
    float wgt[ATT_WARPS];
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) {
        wgt[w] = m_s[w] == -INFINITY ? 0.f : expf(m_s[w] - M);
        L = fmaf(l_s[w], wgt[w], L);
    }
    T* orow = out + ((size_t)t * H + h) * vd;
    for (int d = threadIdx.x; d < vd; d += blockDim.x) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) o = fmaf(acc_s[w * vd + d], wgt[w], o);
        orow[d] = from_f32<T>(o / L);
    }
}

// Rows [t0, t0 + TQ) of the step and one head; rows of one sequence at neighbouring positions are worked together.
__device__ __forceinline__ void att_copy16(float* dst, const float* src, bool live) {            // not live: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
template <int PL, int TQ>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_simt_tile_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, const float* __restrict__ k_cache,
                           const float* __restrict__ v_cache, const int* __restrict__ block_table, int blocks_per_seq,
                           const int* __restrict__ positions, const int* __restrict__ token_slot, int n_tokens, int H, int KV, int hd,
                           float scale, int vd, int v_ld, const float* __restrict__ sink) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kld = hd + 4, vld = vd + 4;            // an odd number of 16-byte pieces a row where hd is a multiple of eight
    float* q_s = smem;                               // [TQ][hd]
    float* m_s = q_s + TQ * hd;                      // [ATT_WARPS][TQ]
    float* l_s = m_s + ATT_WARPS * TQ;
    float* acc_s = l_s + ATT_WARPS * TQ;             // [ATT_WARPS][TQ][vd]
    float* k_s = acc_s + ATT_WARPS * TQ * vd + warp * 32 * (kld + vld);      // the warp's chunk: [32][kld], [32][vld]
    float* v_s = k_s + 32 * kld;
    float* p_s = acc_s + ATT_WARPS * TQ * vd + ATT_WARPS * 32 * (kld + vld) + warp * TQ * 32;
    const int t0 = (gridDim.x - 1 - blockIdx.x) * TQ, t1 = min(t0 + TQ, n_tokens), h = blockIdx.y;      // the last rows see the most keys
    const int g = h / (H / KV);
    for (int a = t0; a < t1;) {
        const int slot = token_slot[a], pos0 = positions[a];
        int n = 1;                                   // rows of this run
        while (a + n < t1 && token_slot[a + n] == slot && positions[a + n] == pos0 + n) ++n;
        if (slot < 0) { a += n; continue; }          // padding rows: nothing is written
        __syncthreads();                             // the run before is done with shared memory
        for (int i = threadIdx.x; i < n * hd; i += ATT_WARPS * 32) q_s[i] = q[(size_t)(a + i / hd) * q_stride + (size_t)h * hd + i % hd];
        __syncthreads();
        const int* table = block_table + (size_t)slot * blocks_per_seq;
        float m[TQ], l[TQ], acc[TQ][PL];
#pragma unroll
        for (int r = 0; r < TQ; ++r) {
            m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
            for (int i = 0; i < PL; ++i) acc[r][i] = 0.f;
        }
        const int last = pos0 + n - 1;
        for (int c = warp; c * 32 <= last; c += ATT_WARPS) {
            const int base = c * 32;
            const size_t row = ((size_t)table[base / PAGE] * KV + g) * PAGE + base % PAGE;
            for (int e = lane; e < 32 * (hd / 4); e += 32) {
                const int j = e / (hd / 4), x = (e - j * (hd / 4)) * 4;
                att_copy16(k_s + j * kld + x, k_cache + (row + j) * hd + x, base + j <= last);
            }
            for (int e = lane; e < 32 * (vd / 4); e += 32) {
                const int j = e / (vd / 4), x = (e - j * (vd / 4)) * 4;
                att_copy16(v_s + j * vld + x, v_cache + (row + j) * v_ld + x, base + j <= last);
            }
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
            __syncwarp();
            const int key = base + lane;
            float s[TQ];
#pragma unroll
            for (int r = 0; r < TQ; ++r) s[r] = 0.f;
            for (int x = 0; x < hd; x += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(k_s + lane * kld + x);
#pragma unroll
                for (int r = 0; r < TQ; ++r) s[r] += dot4(kv, *reinterpret_cast<const float4*>(q_s + (r < n ? r : 0) * hd + x));
            }
#pragma unroll
            for (int r = 0; r < TQ; ++r) {
                if (r >= n || base > pos0 + r) continue;             // the chunk holds no key of this row
                const bool valid = key <= pos0 + r;
                const float sr = valid ? s[r] * scale : -INFINITY;
                const float m_new = fmaxf(m[r], warp_max(sr));
                const float corr = expf(m[r] - m_new);
                const float p = valid ? expf(sr - m_new) : 0.f;
                l[r] = fmaf(l[r], corr, warp_sum(p));
                m[r] = m_new;
#pragma unroll
                for (int i = 0; i < PL; ++i) acc[r][i] *= corr;
                p_s[r * 32 + lane] = p;
            }
            __syncwarp();
            if (base + 31 <= pos0 && n == TQ) {                      // every row sees all 32 keys
                for (int j = 0; j < 32; j += 4) {
                    float v[4][PL];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int i = 0; i < PL; ++i) v[u][i] = lane + 32 * i < vd ? v_s[(j + u) * vld + lane + 32 * i] : 0.f;
#pragma unroll
                    for (int r = 0; r < TQ; ++r) {
                        const float4 p = *reinterpret_cast<const float4*>(p_s + r * 32 + j);
#pragma unroll
                        for (int i = 0; i < PL; ++i)
                            acc[r][i] = fmaf(p.w, v[3][i], fmaf(p.z, v[2][i], fmaf(p.y, v[1][i], fmaf(p.x, v[0][i], acc[r][i]))));
                    }
                }
            } else {
                for (int j = 0; j <= min(31, last - base); ++j)
#pragma unroll
                    for (int r = 0; r < TQ; ++r) {
                        if (r >= n || base + j > pos0 + r) continue; // a key past a row never meets it, whatever it holds
                        const float p = p_s[r * 32 + j];
#pragma unroll
                        for (int i = 0; i < PL; ++i)
                            if (lane + 32 * i < vd) acc[r][i] = fmaf(p, v_s[j * vld + lane + 32 * i], acc[r][i]);
                    }
            }
            __syncwarp();                                            // the chunk is read before the next one takes its place
        }
#pragma unroll
        for (int r = 0; r < TQ; ++r) {
            if (r >= n) continue;
            if (lane == 0) { m_s[warp * TQ + r] = m[r]; l_s[warp * TQ + r] = l[r]; }
#pragma unroll
            for (int i = 0; i < PL; ++i)
                if (lane + 32 * i < vd) acc_s[(warp * TQ + r) * vd + lane + 32 * i] = acc[r][i];
        }
        __syncthreads();
        for (int r = warp; r < n; r += ATT_WARPS) {
            float M = m_s[r];
#pragma unroll
            for (int w = 1; w < ATT_WARPS; ++w) M = fmaxf(M, m_s[w * TQ + r]);
            const float snk = sink ? sink[h] : -INFINITY;
            M = fmaxf(M, snk);
            float L = sink ? expf(snk - M) : 0.f;
            float wgt[ATT_WARPS];
#pragma unroll
            for (int w = 0; w < ATT_WARPS; ++w) {
                wgt[w] = m_s[w * TQ + r] == -INFINITY ? 0.f : expf(m_s[w * TQ + r] - M);
                L = fmaf(l_s[w * TQ + r], wgt[w], L);
            }
            for (int d = lane; d < vd; d += 32) {
                float o = 0.f;
#pragma unroll
                for (int w = 0; w < ATT_WARPS; ++w) o = fmaf(acc_s[(w * TQ + r) * vd + d], wgt[w], o);
                out[((size_t)(a + r) * H + h) * vd + d] = o / L;
            }
        }
        a += n;
    }
}

static size_t simt_tile_smem(int TQ, int hd, int vd) {
    return (size_t)(TQ * hd + 2 * ATT_WARPS * TQ + ATT_WARPS * TQ * vd + ATT_WARPS * 32 * (hd + vd + 8) + ATT_WARPS * TQ * 32) * sizeof(float);
}

// Rows of a tile: 8, 1, or 0 for the row kernel.  us with the row kernel / one row a tile / eight (heads on key heads, size of keys):
//   eight, a prompt of many keys whose tiles give most SMs a CTA (fewer when heads are long):
//     777 tokens, 32 on 8 of 64 757 / - / 480, of 128 1,409 / - / 1,009, 6 on 2 of 32 99 / - / 68; 64 tokens after 1,000, 32 on 8 of 64 168 / - / 98;
//     but 16 tokens after 500 of 8 on 2 of 64 22 / - / 46, 8 prompts of 128 of 32 on 8 203 / - / 259, heads of 16 never
//   one, where every CTA is resident at once: a decode step finds its keys in memory, not in a cache, and a tile has a chunk's keys and values
//   on their way together, the row kernel one batch after another (a step of one sequence of 300 keys through two layers of width 2,048:
//   191 us by rows, 182 by tiles):
//     8 tokens of 300 keys, 32 on 8 of 64 22 / 16 / -; 64 of 1,500 keys, 8 on 2 of 64 106 / 60 / -; 16 after 500, 12 on 4 of 96 46 / 31 / -;
//     but a prompt of five, 32 on 8 of 64 4.0 / 5.6 / - (runs < 0: few keys), and, with more CTAs, 64 tokens of 20 keys 10.4 / 30 / -
static int simt_rows_of_a_tile(int n_tokens, int H, int hd, int vd, int runs) {
    const int sms = sm_count();
    if (sms <= 0 || runs < 0) return 0;
    const long long rows = (long long)n_tokens * H, tiles = (long long)(n_tokens + 7) / 8 * H;
    if (runs > 0 && hd >= 32 && tiles >= (hd > 64 ? 64 : sms)) return 8;
    const long long resident = (228 * 1024) / (long long)(simt_tile_smem(1, hd, vd) + 1024);       // CTAs that an SM's shared memory holds
    return rows <= resident * sms ? 1 : 0;
}

template <int PL, int TQ>
static int launch_simt_tiles(const float* q, int q_stride, float* out, const float* k_cache, const float* v_cache, const int* block_table,
                             int blocks_per_seq, const int* positions, const int* token_slot, int n_tokens, int H, int KV, int hd, float scale,
                             int vd, int v_ld, const float* sink, cudaStream_t stream) {
    const size_t smem = simt_tile_smem(TQ, hd, vd);
    KL_CUDA(cudaFuncSetAttribute(attention_simt_tile_kernel<PL, TQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_kernel(attention_simt_tile_kernel<PL, TQ>, dim3((n_tokens + TQ - 1) / TQ, H), ATT_WARPS * 32, smem, stream, q, q_stride, out, k_cache, v_cache,
                  block_table, blocks_per_seq, positions, token_slot, n_tokens, H, KV, hd, scale, vd, v_ld, sink);
    KL_LAUNCH_CHECK();
    return KL_OK;
}

}  // namespace kl

using namespace kl;

// q: rows of q_stride elements, head h at column h * hd.  out: [tokens, H * vd].  vd <= 0 means values like
// keys (vd = v_ld = hd).  sink: float32 [H] or null.  chunk: positions per chunk (0: none).  rel: float32 [H, rel_n] or null.
// runs: 1, most rows follow the row before them in the same sequence and read hundreds of keys (a long prompt); -1, no row reads more
// than a few dozen keys; 0, unknown.  The results are the same.
KL_API int kl_attention_simt(const void* q, int q_stride, void* out, const void* k_cache, const void* v_cache,
                             const int* block_table, int blocks_per_seq, const int* positions,
                             const int* token_slot, int n_tokens, int H, int KV, int hd, float scale, int window,
                             int vd, int v_ld, const float* sink, int chunk, const float* rel, int rel_n, int runs, int dtype,
                             cudaStream_t stream) {
    if (n_tokens <= 0) return KL_OK;
    if (vd <= 0) { vd = hd; v_ld = hd; }
    if (vd > ATT_MAX_VALUE_DIM || hd <= 0 || v_ld < vd || KV <= 0 || H % KV) return KL_ERR_BAD_SIZE;
    if (H > 65535 || chunk < 0 || (rel != nullptr && rel_n < 1)) return KL_ERR_BAD_SIZE;
    if (dtype == KL_F32 && window <= 0 && chunk == 0 && rel == nullptr && hd % 4 == 0 && vd % 4 == 0 && v_ld % 4 == 0 && hd <= 128 && vd <= 128 &&
        ((uintptr_t)k_cache | (uintptr_t)v_cache) % 16 == 0) {
#define KL_TILES(PL, TQ)                                                                                                                   \
    launch_simt_tiles<PL, TQ>((const float*)q, q_stride, (float*)out, (const float*)k_cache, (const float*)v_cache, block_table, blocks_per_seq, \
                              positions, token_slot, n_tokens, H, KV, hd, scale, vd, v_ld, sink, stream)
        const int tq = simt_rows_of_a_tile(n_tokens, H, hd, vd, runs);
        if (tq == 8) return vd <= 64 ? KL_TILES(2, 8) : KL_TILES(4, 8);
        if (tq == 1) return vd <= 64 ? KL_TILES(2, 1) : KL_TILES(4, 1);
#undef KL_TILES
    }
    const dim3 grid(n_tokens, H);
    const size_t smem = (size_t)(hd + 2 * ATT_WARPS + ATT_WARPS * vd) * sizeof(float);
    if (smem > 200 * 1024) return KL_ERR_BAD_SIZE;
#define KL_ATT(T, PL)                                                                                                         \
    do {                                                                                                                      \
        if (smem > 48 * 1024) KL_CUDA(cudaFuncSetAttribute(attention_simt_kernel<T, PL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        launch_kernel(attention_simt_kernel<T, PL>, grid, ATT_WARPS * 32, smem, stream, (const T*)q, q_stride, (T*)out,       \
                      (const T*)k_cache, (const T*)v_cache, block_table, blocks_per_seq, positions, token_slot, H, KV, hd,    \
                      scale, window, vd, v_ld, sink, chunk, rel, rel_n);                                                                         \
    } while (0)
#define KL_ATT_T(T)                                                                                                           \
    do {                                                                                                                      \
        if (vd <= 64) KL_ATT(T, 2); else if (vd <= 128) KL_ATT(T, 4); else if (vd <= 256) KL_ATT(T, 8); else KL_ATT(T, 16);   \
    } while (0)
    if (dtype == KL_F32) KL_ATT_T(float);
    else if (dtype == KL_BF16) KL_ATT_T(bf16);
    else return KL_ERR_BAD_DTYPE;
#undef KL_ATT_T
#undef KL_ATT
    KL_LAUNCH_CHECK();
    return KL_OK;
}
