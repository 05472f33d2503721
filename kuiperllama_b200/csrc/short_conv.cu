// A short causal convolution over time, one filter per channel, for a ragged step:
//
//   y[t, c] = act( (add_input ? x[t, c] : 0) + bias[c] + sum_j w[c, j] * x[t - (taps - 1) + j, c] )
//
// x before a sequence's first token is zero; x before the step's first token of a sequence that is already
// running comes from the slot's state, which holds the last taps - 1 inputs (oldest first) as [taps - 1, C]
// float32.  Two uses: the convolution in front of a mixer that is added to its own input (output in the
// compute dtype), and the convolution with bias and SiLU over the channels of a state-space mixer (output
// float32, since it enters a recurrence).  The sums run in 32 bits in the order j = 0 .. taps - 1, whatever
// the cut of the prompt, so a result does not depend on the cut.
//
//   short_conv4_kernel        four taps, channels in fours on aligned rows: a thread takes four channels of a tile of tokens and
//                             keeps the last three inputs in registers, so an input is read once per tile (and three times more at
//                             its border) in pieces of four channels, four tokens' pieces in flight.  Bound by bytes: 4,001 tokens of
//                             4,352 channels, bfloat16 in, float32 out (104 MB) 34 us, 128 with a channel a thread.
//   short_conv_kernel         any taps, channels and strides: a CTA per (sequence, tile of tokens), a channel per thread.
//   short_conv_state_kernel   a thread per (sequence, channel): the state after the step.  It runs after the
//                             convolution (stream order), because the convolution's CTAs read the old state.  Where one tile holds
//                             the whole step (a decode step) every channel has one thread, which moves the state on itself.
//
// ExiledOfCode/KuiperLLama has no convolution (its layers are kuiper/source/model/llama3.cpp:146-166).
#include "common.cuh"

namespace kl {

constexpr int SC_MAX_TAPS = 16;
constexpr int SC_TILE = 8;         // tokens per CTA

__device__ __forceinline__ void sc_ld4(const float* p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void sc_ld4(const bf16* p, float (&x)[4]) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    x[0] = __uint_as_float(v.x << 16); x[1] = __uint_as_float(v.x & 0xffff0000u);
    x[2] = __uint_as_float(v.y << 16); x[3] = __uint_as_float(v.y & 0xffff0000u);
}
__device__ __forceinline__ void sc_st4(float* p, const float (&x)[4]) { *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]); }
__device__ __forceinline__ void sc_st4(bf16* p, const float (&x)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x[0], x[1]), b = __floats2bfloat162_rn(x[2], x[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// `move_state`: one tile holds the whole step, and the state moves on here.  `state` rows lie on 16-byte boundaries.
template <typename T, typename TO>
__global__ void __launch_bounds__(256)
short_conv4_kernel(const T* __restrict__ x, long long ld_x, const float* __restrict__ w, const float* __restrict__ bias, float* state,
                   long long ld_state, const int* __restrict__ cu_tokens, const int* __restrict__ seq_slots, int channels, int tile, int add_input,
                   int act_silu, int move_state, TO* __restrict__ out, long long ld_out) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int U = 4;                                         // tokens whose inputs are requested together
    const int s = blockIdx.y;
    const int row0 = cu_tokens[s], n_new = cu_tokens[s + 1] - row0;
    const int first = blockIdx.x * tile, last = min(first + tile, n_new);
    const int c = (blockIdx.z * blockDim.x + threadIdx.x) * 4;
    if (first >= n_new || c >= channels) return;
    float* st = state + (size_t)seq_slots[s] * ld_state + c;
    float wj[4][4], b[4] = {0.f, 0.f, 0.f, 0.f}, win[3][4];      // taps of four channels; the three inputs before the next token
#pragma unroll
    for (int e = 0; e < 4; ++e) sc_ld4(w + (size_t)(c + e) * 4, wj[e]);
    if (bias != nullptr) sc_ld4(bias + c, b);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int li = first - 3 + k;
        if (li >= 0) sc_ld4(x + (size_t)(row0 + li) * ld_x + c, win[k]);
        else sc_ld4(st + (size_t)(3 + li) * channels, win[k]);   // zero in a fresh slot: nothing before the first token
    }
    for (int t0 = first; t0 < last; t0 += U) {
        float in[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) sc_ld4(x + (size_t)(row0 + min(t0 + u, last - 1)) * ld_x + c, in[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (t0 + u >= last) break;
            float y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float acc = wj[e][0] * win[0][e];
                acc = fmaf(wj[e][1], win[1][e], acc);
                acc = fmaf(wj[e][2], win[2][e], acc);
                acc = fmaf(wj[e][3], in[u][e], acc);
                acc += b[e];
                if (add_input) acc += in[u][e];
                y[e] = act_silu ? acc / (1.0f + expf(-acc)) : acc;
                win[0][e] = win[1][e]; win[1][e] = win[2][e]; win[2][e] = in[u][e];
            }
            sc_st4(out + (size_t)(row0 + t0 + u) * ld_out + c, y);
        }
    }
    if (move_state) {
#pragma unroll
        for (int k = 0; k < 3; ++k) sc_st4(st + (size_t)k * channels, win[k]);
    }
}

template <typename T, typename TO>
__global__ void __launch_bounds__(256)
short_conv_kernel(const T* __restrict__ x, long long ld_x, const float* __restrict__ w, const float* __restrict__ bias, int taps,
                  const float* __restrict__ state, long long ld_state, const int* __restrict__ cu_tokens,
                  const int* __restrict__ seq_slots, int channels, int add_input, int act_silu, TO* __restrict__ out, long long ld_out) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.y;
    const int row0 = cu_tokens[s], n_new = cu_tokens[s + 1] - row0;
    const int first = blockIdx.x * SC_TILE;
    if (first >= n_new) return;
    const int last = min(first + SC_TILE, n_new);
    const int slot = seq_slots[s];
    const float* st = state + (size_t)slot * ld_state;
    for (int c = blockIdx.z * blockDim.x + threadIdx.x; c < channels; c += gridDim.z * blockDim.x) {
        float wj[SC_MAX_TAPS];
#pragma unroll
        for (int j = 0; j < SC_MAX_TAPS; ++j) wj[j] = j < taps ? w[(size_t)c * taps + j] : 0.f;
        const float b = bias != nullptr ? bias[c] : 0.f;
        for (int t = first; t < last; ++t) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < SC_MAX_TAPS; ++j) {
                if (j < taps) {
                    const int li = t - (taps - 1) + j;              // index among the step's tokens of this sequence
                    float v;
                    if (li >= 0) v = to_f32(x[(size_t)(row0 + li) * ld_x + c]);
                    else v = st[(size_t)(taps - 1 + li) * channels + c];   // zero in a fresh slot: nothing before the first token
                    acc = fmaf(wj[j], v, acc);
                }
            }
            float y = acc + b;
            if (add_input) y += to_f32(x[(size_t)(row0 + t) * ld_x + c]);
            if (act_silu) y = y / (1.0f + expf(-y));
            out[(size_t)(row0 + t) * ld_out + c] = from_f32<TO>(y);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
short_conv_state_kernel(const T* __restrict__ x, long long ld_x, int taps, float* __restrict__ state, long long ld_state,
                        const int* __restrict__ cu_tokens, const int* __restrict__ seq_slots, int channels) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.y;
    const int row0 = cu_tokens[s], n_new = cu_tokens[s + 1] - row0;
    if (n_new <= 0) return;
    float* st = state + (size_t)seq_slots[s] * ld_state;
    const int keep = taps - 1;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < channels; c += gridDim.x * blockDim.x) {
        float next[SC_MAX_TAPS];
#pragma unroll
        for (int k = 0; k < SC_MAX_TAPS; ++k) {
            if (k < keep) {
                const int li = n_new - keep + k;
                next[k] = li >= 0 ? to_f32(x[(size_t)(row0 + li) * ld_x + c]) : st[(size_t)(keep + li) * channels + c];
            }
        }
#pragma unroll
        for (int k = 0; k < SC_MAX_TAPS; ++k)
            if (k < keep) st[(size_t)k * channels + c] = next[k];
    }
}

}  // namespace kl

using namespace kl;

// The state alone after a step (a caller whose own kernel convolved): the last taps - 1 rows of x, `channels` wide, per sequence.
KL_API int kl_short_conv_state(const void* x, long long ld_x, int taps, float* state, long long ld_state, const int* cu_tokens,
                               const int* seq_slots, int n_seqs, int channels, int dtype, cudaStream_t stream) {
    if (n_seqs <= 0 || channels <= 0 || taps <= 1) return KL_OK;
    if (taps > SC_MAX_TAPS || n_seqs > 65535) return KL_ERR_BAD_SIZE;
    const int threads = channels >= 256 ? 256 : ((channels + 31) / 32) * 32;
    const dim3 grid((channels + threads - 1) / threads, n_seqs);
    if (dtype == KL_F32)
        launch_kernel(short_conv_state_kernel<float>, grid, threads, 0, stream, (const float*)x, ld_x, taps, state, ld_state, cu_tokens, seq_slots, channels);
    else if (dtype == KL_BF16)
        launch_kernel(short_conv_state_kernel<bf16>, grid, threads, 0, stream, (const bf16*)x, ld_x, taps, state, ld_state, cu_tokens, seq_slots, channels);
    else
        return KL_ERR_BAD_DTYPE;
    KL_LAUNCH_CHECK();
    return KL_OK;
}

// x: compute dtype `dtype`; out: float32 if out_f32 else the compute dtype.  state: float32, the slot's row starts at
// state + slot * ld_state and holds [taps - 1, channels].  With update_state the state moves on in a second launch.
KL_API int kl_short_conv(const void* x, long long ld_x, const float* w, const float* bias, int taps, float* state, long long ld_state,
                         const int* cu_tokens, const int* seq_slots, int n_seqs, int max_new, int channels, int add_input,
                         int act_silu, void* out, long long ld_out, int out_f32, int update_state, int dtype, cudaStream_t stream) {
    if (n_seqs <= 0 || max_new <= 0 || channels <= 0) return KL_OK;
    if (taps < 1 || taps > SC_MAX_TAPS) return KL_ERR_BAD_SIZE;
    if (dtype != KL_F32 && dtype != KL_BF16) return KL_ERR_BAD_DTYPE;
    const size_t es = dtype == KL_F32 ? 4 : 2, os = out_f32 || dtype == KL_F32 ? 4 : 2;
    if (taps == 4 && channels % 4 == 0 && ld_x % 4 == 0 && ld_out % 4 == 0 && ld_state % 4 == 0 && (uintptr_t)x % (4 * es) == 0 &&
        (uintptr_t)out % (4 * os) == 0 && ((uintptr_t)w | (uintptr_t)state | (uintptr_t)bias) % 16 == 0 && n_seqs <= 65535) {
        // tiles of 16 tokens, shorter ones while the device would have fewer than 16 warps an SM
        const int threads = channels / 4 >= 128 ? 128 : (channels / 4 + 31) / 32 * 32, zblocks = (channels / 4 + threads - 1) / threads;
        int tile = 16;
        while (tile > 4 && (long long)((max_new + tile - 1) / tile) * n_seqs * zblocks * (threads / 32) < 16LL * sm_count()) tile >>= 1;
        const int tiles = (max_new + tile - 1) / tile, moves = update_state && tiles == 1;
        const dim3 grid(tiles, n_seqs, zblocks);
#define KL_SC4(T, TO)                                                                                                         \
    launch_kernel(short_conv4_kernel<T, TO>, grid, threads, 0, stream, (const T*)x, ld_x, w, bias, state, ld_state, cu_tokens, seq_slots, channels, \
                  tile, add_input, act_silu, moves, (TO*)out, ld_out)
        if (dtype == KL_F32) KL_SC4(float, float);
        else if (out_f32) KL_SC4(bf16, float);
        else KL_SC4(bf16, bf16);
#undef KL_SC4
        KL_LAUNCH_CHECK();
        if (!update_state || moves) return KL_OK;
        return kl_short_conv_state(x, ld_x, taps, state, ld_state, cu_tokens, seq_slots, n_seqs, channels, dtype, stream);
    }
    const int threads = channels >= 256 ? 256 : ((channels + 31) / 32) * 32;
    const int tiles = (max_new + SC_TILE - 1) / SC_TILE;
    int zblocks = (channels + threads - 1) / threads;
    if (zblocks > 64) zblocks = 64;
    dim3 grid(tiles, n_seqs, zblocks);
#define KL_SC(T, TO)                                                                                                          \
    launch_kernel(short_conv_kernel<T, TO>, grid, threads, 0, stream, (const T*)x, ld_x, w, bias, taps, (const float*)state, ld_state, \
                  cu_tokens, seq_slots, channels, add_input, act_silu, (TO*)out, ld_out)
    if (dtype == KL_F32) KL_SC(float, float);
    else if (out_f32) KL_SC(bf16, float);
    else KL_SC(bf16, bf16);
#undef KL_SC
    KL_LAUNCH_CHECK();
    if (update_state) return kl_short_conv_state(x, ld_x, taps, state, ld_state, cu_tokens, seq_slots, n_seqs, channels, dtype, stream);
    return KL_OK;
}
