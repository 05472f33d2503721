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
// attention_simt_token_kernel does the same for float32 rows without a window, chunks or distance bias (key and value sizes up to 128):
// a warp copies its chunk of keys and values to shared memory first, as whole lines.  attention_simt_prompt_kernel takes such rows of a
// prompt together, several of them and of the heads of one key head, which share the copies.  Every token's sums are the same operations in the
// same order as in the kernel above, so its result has the same bits.  simt_plan says where each of them runs.  What bounds the prompt kernel
// is the issue of its instructions (2.4 a cycle and SM of 4): 84 million for 777 tokens, 32 heads of 64 on 8, of which the sums as they are ordered take
// 50.  131 us; tiles of eight rows whose warps copied their chunks each for themselves and waited for them 480, a CTA per token 750; 2,048 tokens 723 /
// 2,404 / 4,920; 777 of 128 262 / 1,007 / 1,405.
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

__device__ __forceinline__ void att_copy16(float* dst, const float* src, bool live) {            // not live: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
// A row of the step and a head; a warp's chunk of keys and values is on its way together.
template <int PL>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_simt_token_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, const float* __restrict__ k_cache,
                            const float* __restrict__ v_cache, const int* __restrict__ block_table, int blocks_per_seq,
                            const int* __restrict__ positions, const int* __restrict__ token_slot, int H, int KV, int hd, float scale, int vd,
                            int v_ld, const float* __restrict__ sink) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kld = hd + 4, vld = vd + 4;            // an odd number of 16-byte pieces a row where hd is a multiple of eight
    float* q_s = smem;
    float* m_s = q_s + hd;                           // [ATT_WARPS]
    float* l_s = m_s + ATT_WARPS;
    float* acc_s = l_s + ATT_WARPS;                  // [ATT_WARPS][vd]
    float* k_s = acc_s + ATT_WARPS * vd + warp * 32 * (kld + vld);           // the warp's chunk: [32][kld], [32][vld]
    float* v_s = k_s + 32 * kld;
    float* p_s = acc_s + ATT_WARPS * vd + ATT_WARPS * 32 * (kld + vld) + warp * 32;
    const int a = gridDim.x - 1 - blockIdx.x, h = blockIdx.y, g = h / (H / KV);
    const int slot = token_slot[a], pos = positions[a];
    if (slot < 0) return;                            // a padding row: nothing is written
    for (int i = threadIdx.x; i < hd; i += ATT_WARPS * 32) q_s[i] = q[(size_t)a * q_stride + (size_t)h * hd + i];
    __syncthreads();
    const int* table = block_table + (size_t)slot * blocks_per_seq;
    float m = -INFINITY, l = 0.f, acc[PL];
#pragma unroll
    for (int i = 0; i < PL; ++i) acc[i] = 0.f;
    for (int c = warp; c * 32 <= pos; c += ATT_WARPS) {
        const int base = c * 32;
        const size_t row = ((size_t)table[base / PAGE] * KV + g) * PAGE + base % PAGE;
        for (int e = lane; e < 32 * (hd / 4); e += 32) {
            const int j = e / (hd / 4), x = (e - j * (hd / 4)) * 4;
            att_copy16(k_s + j * kld + x, k_cache + (row + j) * hd + x, base + j <= pos);
        }
        for (int e = lane; e < 32 * (vd / 4); e += 32) {
            const int j = e / (vd / 4), x = (e - j * (vd / 4)) * 4;
            att_copy16(v_s + j * vld + x, v_cache + (row + j) * v_ld + x, base + j <= pos);
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        float s = 0.f;
        for (int x = 0; x < hd; x += 4) s += dot4(*reinterpret_cast<const float4*>(k_s + lane * kld + x), *reinterpret_cast<const float4*>(q_s + x));
        const bool valid = base + lane <= pos;
        const float sr = valid ? s * scale : -INFINITY;
        const float m_new = fmaxf(m, warp_max(sr));
        const float corr = expf(m - m_new);
        const float p = valid ? expf(sr - m_new) : 0.f;
        l = fmaf(l, corr, warp_sum(p));
        m = m_new;
#pragma unroll
        for (int i = 0; i < PL; ++i) acc[i] *= corr;
        p_s[lane] = p;
        __syncwarp();
        if (base + 31 <= pos) {                      // all 32 keys are seen
            for (int j = 0; j < 32; j += 4) {
                const float4 w = *reinterpret_cast<const float4*>(p_s + j);
#pragma unroll
                for (int i = 0; i < PL; ++i) {
                    const float* v = v_s + j * vld + lane + 32 * i;
                    if (lane + 32 * i < vd) acc[i] = fmaf(w.w, v[3 * vld], fmaf(w.z, v[2 * vld], fmaf(w.y, v[vld], fmaf(w.x, v[0], acc[i]))));
                }
            }
        } else {                                     // (a key past the row never meets it, whatever it holds)
            for (int j = 0; j <= pos - base; ++j)
#pragma unroll
                for (int i = 0; i < PL; ++i)
                    if (lane + 32 * i < vd) acc[i] = fmaf(p_s[j], v_s[j * vld + lane + 32 * i], acc[i]);
        }
        __syncwarp();                                // the chunk is read before the next one takes its place
    }
    if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
#pragma unroll
    for (int i = 0; i < PL; ++i)
        if (lane + 32 * i < vd) acc_s[warp * vd + lane + 32 * i] = acc[i];
    __syncthreads();
    if (warp != 0) return;
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
    for (int d = lane; d < vd; d += 32) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) o = fmaf(acc_s[w * vd + d], wgt[w], o);
        out[((size_t)a * H + h) * vd + d] = o / L;
    }
}

// For prompts of many keys: sixteen warps and one key head.  Unit u of the four has 4 R rows of one of its heads (`hb` heads: as many as share the keys,
// four, two or one; the units beyond take the rows further on); the chunks of 32 keys, dealt to four classes as in the kernels above, are copied
// once for the four units, a class's warps waiting for one another alone: the values arrive while the scores are worked, the next keys while the
// values are.  A lane has R rows r = rr * 4 + lane / 8 and in the scores keys lane % 8 + 8 i, in the values columns (lane % 8) * 4 + 32 i: a maximum and a
// sum of 32 keys are three exchanges, the sum in the order of warp_sum (keys 16 apart, 8 apart, ..).
template <int R, int NV>
__global__ void __launch_bounds__(512)
attention_simt_prompt_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, const float* __restrict__ k_cache,
                             const float* __restrict__ v_cache, const int* __restrict__ block_table, int blocks_per_seq,
                             const int* __restrict__ positions, const int* __restrict__ token_slot, int n_tokens, int H, int KV, int hd,
                             float scale, int vd, int v_ld, const float* __restrict__ sink, int hb) {
    constexpr int TQ = 4 * R, PLD = 40;              // floats of a row of weights: four rows on 32 banks
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, unit = warp & 3, cls = warp >> 2, rg = lane >> 3, k8 = lane & 7;
    const int kld = hd + 4, vld = vd + 4, qld = ((hd + 31) & ~31) + 8;
    float* k_s = smem + cls * 32 * (kld + vld);      // the class's chunk: [32][kld], [32][vld]
    float* v_s = k_s + 32 * kld;
    float* acc_s = smem;                             // in the end: [unit][class][TQ][vd]
    const int tiles = 4 * 32 * (kld + vld), sums = 16 * TQ * vd;
    float* p_s = smem + (tiles > sums ? tiles : sums) + warp * TQ * PLD;
    float* q_s = smem + (tiles > sums ? tiles : sums) + 16 * TQ * PLD;       // [unit][TQ][qld]
    float* m_s = q_s + 4 * TQ * qld;                 // [unit][class][TQ]
    float* l_s = m_s + 16 * TQ;
    const int span = TQ * (4 / hb), ub = unit / hb;
    const int t0 = (gridDim.y - 1 - blockIdx.y) * span, t1 = min(t0 + span, n_tokens);       // the last rows see the most keys: they start first
    const int h0 = blockIdx.x * hb, h = h0 + unit % hb, g = h0 / (H / KV);
    for (int a = t0; a < t1;) {
        const int slot = token_slot[a], pos0 = positions[a];
        int n = 0;                                   // rows of this run
        for (int z = 0; z < span; z += 32) {
            const int r = a + z + lane;
            const unsigned same = __ballot_sync(0xffffffffu, r < t1 && token_slot[min(r, t1 - 1)] == slot && positions[min(r, t1 - 1)] == pos0 + z + lane);
            n += same == 0xffffffffu ? 32 : __ffs(~same) - 1;
            if (same != 0xffffffffu) break;
        }
        if (slot < 0) { a += n; continue; }          // padding rows: nothing is written
        __syncthreads();                             // the run before is done with shared memory
        for (int i = threadIdx.x >> 3; i < 4 * TQ; i += 64) {                // eight threads a row (one past the run: zeros)
            const int u = i / TQ, r = u / hb * TQ + i % TQ;
            const float* src = q + (size_t)(a + min(r, n - 1)) * q_stride + (size_t)(h0 + u % hb) * hd;
            for (int x = threadIdx.x & 7; x < hd; x += 8)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(q_s + i * qld + x)), "l"(src + x),
                             "r"(r < n ? 4 : 0) : "memory");
        }
        const int* table = block_table + (size_t)slot * blocks_per_seq;
        const int rows = min(TQ, n - ub * TQ), pos_u = pos0 + ub * TQ, last_u = pos_u + rows - 1;        // of this unit (none: rows <= 0)
        const int last = pos0 + n - 1;
        float m[R], l[R], acc[R][4 * NV];
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
            m[rr] = -INFINITY; l[rr] = 0.f;
#pragma unroll
            for (int i = 0; i < 4 * NV; ++i) acc[rr][i] = 0.f;
        }
        auto row_of = [&](int c) { return c * 32 <= last ? ((size_t)table[c * 32 / PAGE] * KV + g) * PAGE + c * 32 % PAGE : 0; };
        const int cj = unit * 8 + rg * 2 + (k8 >> 2), cx = (k8 & 3) * 4;     // the row and the first column that this thread copies
        auto copy = [&](float* dst, const float* src, int ld_dst, int ld_src, int width, size_t row, int c) {
            for (int x = cx; x < width; x += 16) att_copy16(dst + cj * ld_dst + x, src + (row + cj) * ld_src + x, c * 32 + cj <= last);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto meet = [&]() { asm volatile("cp.async.wait_group 0;\n\tbar.sync %0, 128;" ::"r"(1 + cls) : "memory"); };
        size_t row = row_of(cls);
        if (cls * 32 <= last) copy(k_s, k_cache, kld, hd, hd, row, cls);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                             // the queries are there
        for (int c = cls; c * 32 <= last; c += 4) {
            const int base = c * 32;
            const bool work = rows > 0 && base <= last_u;
            meet();                                  // the keys are there, everybody is done with the values before
            copy(v_s, v_cache, vld, v_ld, vd, row, c);
            row = row_of(c + 4);
            if (work) {
                float s[R][4];
#pragma unroll
                for (int rr = 0; rr < R; ++rr) s[rr][0] = s[rr][1] = s[rr][2] = s[rr][3] = 0.f;
#pragma unroll 2
                for (int x = 0; x < hd; x += 4) {
                    float4 kv[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) kv[i] = *reinterpret_cast<const float4*>(k_s + (k8 + 8 * i) * kld + x);
#pragma unroll
                    for (int rr = 0; rr < R; ++rr) {
                        const float4 qv = *reinterpret_cast<const float4*>(q_s + (unit * TQ + rr * 4 + rg) * qld + x);
#pragma unroll
                        for (int i = 0; i < 4; ++i) s[rr][i] += dot4(kv[i], qv);
                    }
                }
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
                    const int r = rr * 4 + rg, pos = pos_u + r;
                    const bool on = r < rows && base <= pos;                 // (else the chunk holds no key of this row)
                    bool valid[4];
                    float p[4], mx = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        valid[i] = on && base + k8 + 8 * i <= pos;
                        s[rr][i] = valid[i] ? s[rr][i] * scale : -INFINITY;
                        mx = fmaxf(mx, s[rr][i]);
                    }
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    const float m_new = fmaxf(m[rr], mx);
                    const float corr = on ? expf(m[rr] - m_new) : 1.f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        p[i] = valid[i] ? expf(s[rr][i] - m_new) : 0.f;
                        p_s[r * PLD + k8 + 8 * i] = p[i];
                    }
                    float sum = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    l[rr] = on ? fmaf(l[rr], corr, sum) : l[rr];
                    m[rr] = on ? m_new : m[rr];
#pragma unroll
                    for (int i = 0; i < 4 * NV; ++i) acc[rr][i] *= corr;
                }
            }
            meet();                                  // the values are there, everybody is done with the keys
            if (c * 32 + 128 <= last) copy(k_s, k_cache, kld, hd, hd, row, c + 4);
            if (work) {
                if (base + 31 <= pos_u && rows == TQ) {                      // every row sees all 32 keys
#pragma unroll 2
                    for (int j = 0; j < 32; j += 4) {
                        float4 p[R];
#pragma unroll
                        for (int rr = 0; rr < R; ++rr) p[rr] = *reinterpret_cast<const float4*>(p_s + (rr * 4 + rg) * PLD + j);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int i = 0; i < NV; ++i) {
                                if (k8 * 4 + 32 * i >= vd) continue;
                                const float4 v = *reinterpret_cast<const float4*>(v_s + (j + u) * vld + k8 * 4 + 32 * i);
#pragma unroll
                                for (int rr = 0; rr < R; ++rr) {
                                    const float w = u == 0 ? p[rr].x : u == 1 ? p[rr].y : u == 2 ? p[rr].z : p[rr].w;
                                    acc[rr][4 * i] = fmaf(w, v.x, acc[rr][4 * i]);
                                    acc[rr][4 * i + 1] = fmaf(w, v.y, acc[rr][4 * i + 1]);
                                    acc[rr][4 * i + 2] = fmaf(w, v.z, acc[rr][4 * i + 2]);
                                    acc[rr][4 * i + 3] = fmaf(w, v.w, acc[rr][4 * i + 3]);
                                }
                            }
                    }
                } else {
                    int most[R];                     // the last key of a row in the chunk: a key past it never meets the row, whatever it holds
#pragma unroll
                    for (int rr = 0; rr < R; ++rr) most[rr] = rr * 4 + rg < rows ? pos_u + rr * 4 + rg - base : -1;
#pragma unroll 2
                    for (int j = 0; j <= min(31, last_u - base); j += 4) {
                        float4 p[R];
#pragma unroll
                        for (int rr = 0; rr < R; ++rr) p[rr] = *reinterpret_cast<const float4*>(p_s + (rr * 4 + rg) * PLD + j);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int i = 0; i < NV; ++i) {
                                if (k8 * 4 + 32 * i >= vd) continue;
                                const float4 v = *reinterpret_cast<const float4*>(v_s + (j + u) * vld + k8 * 4 + 32 * i);
#pragma unroll
                                for (int rr = 0; rr < R; ++rr) {
                                    const float w = u == 0 ? p[rr].x : u == 1 ? p[rr].y : u == 2 ? p[rr].z : p[rr].w;
                                    if (j + u > most[rr]) continue;
                                    acc[rr][4 * i] = fmaf(w, v.x, acc[rr][4 * i]);
                                    acc[rr][4 * i + 1] = fmaf(w, v.y, acc[rr][4 * i + 1]);
                                    acc[rr][4 * i + 2] = fmaf(w, v.z, acc[rr][4 * i + 2]);
                                    acc[rr][4 * i + 3] = fmaf(w, v.w, acc[rr][4 * i + 3]);
                                }
                            }
                    }
                }
            }
        }
        __syncthreads();                             // the classes' sums take the place of the keys and values
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
            const int at = (unit * 4 + cls) * TQ + rr * 4 + rg;
            if (k8 == 0) { m_s[at] = m[rr]; l_s[at] = l[rr]; }
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (k8 * 4 + 32 * i < vd)
                    *reinterpret_cast<float4*>(acc_s + at * vd + k8 * 4 + 32 * i) = make_float4(acc[rr][4 * i], acc[rr][4 * i + 1], acc[rr][4 * i + 2], acc[rr][4 * i + 3]);
        }
        __syncthreads();
        for (int r = cls; r < rows; r += ATT_WARPS) {
            const float* mu = m_s + unit * 4 * TQ + r;
            float M = mu[0];
#pragma unroll
            for (int w = 1; w < ATT_WARPS; ++w) M = fmaxf(M, mu[w * TQ]);
            const float snk = sink ? sink[h] : -INFINITY;
            M = fmaxf(M, snk);
            float L = sink ? expf(snk - M) : 0.f;
            float wgt[ATT_WARPS];
#pragma unroll
            for (int w = 0; w < ATT_WARPS; ++w) {
                wgt[w] = mu[w * TQ] == -INFINITY ? 0.f : expf(mu[w * TQ] - M);
                L = fmaf(l_s[(unit * 4 + w) * TQ + r], wgt[w], L);
            }
            for (int d = lane; d < vd; d += 32) {
                float o = 0.f;
#pragma unroll
                for (int w = 0; w < ATT_WARPS; ++w) o = fmaf(acc_s[((unit * 4 + w) * TQ + r) * vd + d], wgt[w], o);
                out[((size_t)(a + ub * TQ + r) * H + h) * vd + d] = o / L;
            }
        }
        a += n;
    }
}
static size_t simt_prompt_smem(int R, int hd, int vd) {
    const int TQ = 4 * R, tiles = 4 * 32 * (hd + vd + 8), sums = 16 * TQ * vd;
    return (size_t)((tiles > sums ? tiles : sums) + 16 * TQ * 40 + 4 * TQ * (((hd + 31) & ~31) + 8) + 32 * TQ) * sizeof(float);
}

static size_t simt_token_smem(int hd, int vd) {
    return (size_t)(hd + 2 * ATT_WARPS + ATT_WARPS * vd + ATT_WARPS * 32 * (hd + vd + 8) + ATT_WARPS * 32) * sizeof(float);
}
// heads of one key head that a CTA of the prompt kernel takes, and the rows that its units then span with R rows a lane
static int simt_heads_together(int H, int KV) { const int per = H / KV; return per % 4 == 0 ? 4 : per % 2 == 0 ? 2 : 1; }
static int simt_span(int R, int hb) { return 4 * R * (4 / hb); }

// Which kernel: 4, 2 or 1 rows a lane of the prompt kernel, -1 the kernel of a row and a head, 0 the row kernel.  `runs`: rows that follow one
// another in a sequence, on average (0 unknown; negative: so many, of a few dozen keys at most).  us with the row kernel / 1 / 2 / 4 rows a lane
// (heads on key heads, size of keys):
//   the prompt kernel where the runs fill a CTA's rows and there are enough CTAs of one row a lane (a chunk of 32 keys takes a CTA about 5 us and its start 4;
//   the row kernel spreads few rows over more CTAs): 64 after 1,500, 32 on 8 of 64 (128 CTAs) 246 / 81 / 111 / 158; 32 after 500 (64) 47 / 31 / 42 /
//   60; 16 after 500 (32) 29 / 31 / 41 / 59; 8 after 500 (16) 23 / 28 / 39 / 51; 16 after 500 of 128 (32) 67 / 51 / 71 / 116, 8 (16) 39 / 49 / 67 / 109;
//   of few keys 8 runs of 16, 16 on 4 of 64 (128) 9.2 / 6.2 / 7.3 / 11, 8 on 2 (64) 5.4 / 6.2 / 7.2 / 11; runs of eight where a CTA spans 16, 8 on 8 of
//   64 25 / 40 / 119 / 330;
//   one row a lane up to a CTA an SM: 128 after 500, 16 on 4 (128) 98 / 35 / 47 / 67, 32 on 8 (256) 194 / 63 / 47 / 68;
//   four where that leaves more CTAs than SMs and the runs are long: 512, 32 on 8 (256 CTAs) 343 / 113 / 80 / 61, 777 748 / 239 / 169 / 131; 256 (128) 97 /
//   - / 27 / 31, 4 runs of 100 71 / - / 30 / 33;
//   a row and a head in a CTA, where every CTA is resident at once: a decode step finds its keys in memory, not in a cache, and has a chunk's keys and
//   values on their way together, the row kernel one batch after another (a step of one sequence of 300 keys through two layers of width
//   2,048: 191 us by rows, 182 so); row kernel / this: 8 tokens of 300 keys, 32 on 8 of 64 22 / 16; 64 of 1,500 keys, 8 on 2 of 64 106 / 60; 16
//   after 500, 12 on 4 of 96 46 / 31; but a prompt of five, 32 on 8 of 64 4.0 / 5.6 (few keys), and, with more CTAs, 64 tokens of 20 keys 10.4 / 30.
static int simt_plan(int n_tokens, int H, int KV, int hd, int vd, int runs) {
    const int sms = sm_count();
    if (sms <= 0) return 0;
    const int hb = simt_heads_together(H, KV), run = runs < 0 ? -runs : runs;
    auto ctas = [&](int R) { return (long long)((n_tokens + simt_span(R, hb) - 1) / simt_span(R, hb)) * (H / hb); };
    if (hd >= 32 && run >= simt_span(1, hb) && ctas(1) >= (runs < 0 ? 96 : 40) * (hd > 64 ? 2 : 3) / 3) {
        if (ctas(1) <= sms) return 1;
        return run >= 256 && ctas(4) > sms ? 4 : 2;
    }
    if (runs < 0) return 0;
    const long long resident = (228 * 1024) / (long long)(simt_token_smem(hd, vd) + 1024);         // CTAs that an SM's shared memory holds
    return (long long)n_tokens * H <= resident * sms ? -1 : 0;
}

template <int R, int NV>
static int launch_simt_prompt(const float* q, int q_stride, float* out, const float* k_cache, const float* v_cache, const int* block_table,
                              int blocks_per_seq, const int* positions, const int* token_slot, int n_tokens, int H, int KV, int hd, float scale,
                              int vd, int v_ld, const float* sink, cudaStream_t stream) {
    const size_t smem = simt_prompt_smem(R, hd, vd);
    const int hb = simt_heads_together(H, KV), span = simt_span(R, hb);
    KL_CUDA(cudaFuncSetAttribute(attention_simt_prompt_kernel<R, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_kernel(attention_simt_prompt_kernel<R, NV>, dim3(H / hb, (n_tokens + span - 1) / span), 512, smem, stream, q, q_stride, out, k_cache, v_cache,
                  block_table, blocks_per_seq, positions, token_slot, n_tokens, H, KV, hd, scale, vd, v_ld, sink, hb);
    KL_LAUNCH_CHECK();
    return KL_OK;
}
template <int PL>
static int launch_simt_tokens(const float* q, int q_stride, float* out, const float* k_cache, const float* v_cache, const int* block_table,
                              int blocks_per_seq, const int* positions, const int* token_slot, int n_tokens, int H, int KV, int hd, float scale,
                              int vd, int v_ld, const float* sink, cudaStream_t stream) {
    const size_t smem = simt_token_smem(hd, vd);
    KL_CUDA(cudaFuncSetAttribute(attention_simt_token_kernel<PL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_kernel(attention_simt_token_kernel<PL>, dim3(n_tokens, H), ATT_WARPS * 32, smem, stream, q, q_stride, out, k_cache, v_cache, block_table,
                  blocks_per_seq, positions, token_slot, H, KV, hd, scale, vd, v_ld, sink);
    KL_LAUNCH_CHECK();
    return KL_OK;
}

}  // namespace kl

using namespace kl;

// q: rows of q_stride elements, head h at column h * hd.  out: [tokens, H * vd].  vd <= 0 means values like
// keys (vd = v_ld = hd).  sink: float32 [H] or null.  chunk: positions per chunk (0: none).  rel: float32 [H, rel_n] or null.
// runs: rows that follow one another in a sequence, on average (a prompt's do); negative: so many, none of which reads more than a few dozen keys; 0,
// unknown.  The results are the same.
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
#define KL_WITH(launch)                                                                                                                      \
    launch((const float*)q, q_stride, (float*)out, (const float*)k_cache, (const float*)v_cache, block_table, blocks_per_seq, positions, token_slot, \
           n_tokens, H, KV, hd, scale, vd, v_ld, sink, stream)
        const int plan = simt_plan(n_tokens, H, KV, hd, vd, runs);
        if (plan == 4) return vd <= 32 ? KL_WITH((launch_simt_prompt<4, 1>)) : vd <= 64 ? KL_WITH((launch_simt_prompt<4, 2>)) : KL_WITH((launch_simt_prompt<4, 4>));
        if (plan == 2) return vd <= 32 ? KL_WITH((launch_simt_prompt<2, 1>)) : vd <= 64 ? KL_WITH((launch_simt_prompt<2, 2>)) : KL_WITH((launch_simt_prompt<2, 4>));
        if (plan == 1) return vd <= 32 ? KL_WITH((launch_simt_prompt<1, 1>)) : vd <= 64 ? KL_WITH((launch_simt_prompt<1, 2>)) : KL_WITH((launch_simt_prompt<1, 4>));
        if (plan == -1) return vd <= 64 ? KL_WITH(launch_simt_tokens<2>) : KL_WITH(launch_simt_tokens<4>);
#undef KL_WITH
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
