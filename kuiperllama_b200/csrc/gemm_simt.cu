// C[M, N] = A[M, K] * W[N, K]^T with plain 32-bit FMA arithmetic: every size, every
// alignment.  It is the matrix product of the true 32-bit path (no tensor-core mode of any
// kind) and the fallback of the bfloat16 path for shapes that the tensor-core kernel
// refuses (a K whose row stride is no multiple of 16 bytes).
//
// y = W x as in ExiledOfCode/KuiperLLama's matmul_kernel_cu_fp32 (matmul_kernel.cu:6-54):
// weights are [out, in] row-major and there is no bias.  There one CTA reduces one output
// row of a single vector.
//
// One order of additions for every kernel of this file, so that the value of an output does not depend on how many rows M
// the call has or which kernel takes it: K is cut into blocks of 512; a block is one chain of fused multiply-adds in ascending k,
// and the output is the sum of its blocks in ascending order.
//
// * gemm_rows_kernel (few rows of A: a decode step) is bound by reading W once.  A warp takes 8 rows of W and four blocks of K,
//   a lane one row and one block; the warp copies its weights by 16-byte cp.async into a ring of its own, two chunks (17 KB a
//   warp, 70 KB an SM) ahead of the arithmetic, without a break between one set of rows and the next, the first ones before the
//   kernel ahead has finished.  W of 16,384 x 2,048: 30 us for one row of A (4.4 TB/s), 64 for eight (the shared-memory reads
//   of A bind); 2,048 x 2,048 7 and 17 us.
// * gemm_tile_kernel (everything else) is bound by the FMA pipe.  128 threads make a tile of 64 x 128 outputs, 8 x 8 each, as
//   packed pairs of rows of A (fma.rn.f32x2: the same two results in one instruction, whose operands come from both register
//   banks).  A lies in shared memory with the row innermost (4-byte cp.async), W with k innermost (16-byte cp.async); the sums of
//   blocks live in shared memory.  The blocks of K are dealt to a cluster of CTAs where the tiles alone leave multiprocessors
//   idle; its CTAs add each other's sums through distributed shared memory, in order.  Tiles of 64 x 32 where even that is less
//   than three CTAs for two SMs.  777 x 16,384 x 2,048: 1.26 ms (41 TFLOP/s; 72 is what the pipe gives register operands),
//   777 x 2,048 x 8,192: 0.77 ms.
#include <cooperative_groups.h>
#include "common.cuh"

namespace kl {

namespace cg = cooperative_groups;

constexpr int BLOCK = 512;

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? BYTES : 0;                             // 0: the place is filled with zeros
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpair(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// ------------------------------------------------------------------------------------------------ few rows of A

constexpr int GR_WARPS = 4, GR_ROWS = 8, GR_LANES = 4, GR_STAGES = 3, GR_SPAN = GR_LANES * BLOCK;

// A chunk brings CHUNK k of each of a warp's four blocks: of 8 rows of W and of MT rows of A.  Rows of CHUNK + 4 floats are an odd number
// of 16-byte pieces, so eight rows lie on eight bank groups.
template <int MT>
struct Rows {
    static constexpr int CHUNK = MT >= 4 ? 32 : 64, PAD = CHUNK + 4, PER = BLOCK / CHUNK;
    static constexpr int W_FLOATS = GR_LANES * GR_ROWS * PAD, STAGE = W_FLOATS + GR_LANES * MT * PAD;
};

// Warp w of a CTA: rows 8 * (w / wb) .. of an item's 8 * (4 / wb), spans of four blocks w % wb, + wb, ...; lane = row + 8 * block.
// Items (sets of rows) blockIdx.x, + gridDim.x, ...
// FULL: the last span's first block is a whole one, so that every span has the same number of chunks.
template <int MT, bool FULL>
__global__ void __launch_bounds__(GR_WARPS * 32)
gemm_rows_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc,
                 int M, int N, int K, int wb) {
    using R = Rows<MT>;
    pdl_launch_dependents();
    extern __shared__ __align__(16) float gr_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows_item = GR_ROWS * (GR_WARPS / wb), items = (N + rows_item - 1) / rows_item;
    const int my_row = (warp / wb) * GR_ROWS, first = warp % wb;
    const int m0 = blockIdx.y * MT;
    const int nb = (K + BLOCK - 1) / BLOCK, spans = (nb + GR_LANES - 1) / GR_LANES;
    const int mine = first < spans ? (spans - 1 - first) / wb + 1 : 0;        // spans of this warp
    // chunks of a span: the last one stops where its first block does (64 columns of 64 in one chunk: 2 us, 15 with all eight or sixteen)
    const int last_parts = FULL ? R::PER : min(R::PER, (K - (spans - 1) * GR_SPAN + R::CHUNK - 1) / R::CHUNK);
    auto parts = [&](int span) { return FULL || span < spans - 1 ? R::PER : last_parts; };
    float* ring = gr_smem + warp * GR_STAGES * R::STAGE;
    float* sums = gr_smem + GR_WARPS * GR_STAGES * R::STAGE;                  // two of [blocks][MT][rows_item]
    const int sums_floats = spans * GR_LANES * MT * rows_item;
    const int n_items = (int)blockIdx.x < items ? (items - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const int chunks = mine > 0 ? ((mine - 1) * R::PER + parts(first + (mine - 1) * wb)) * n_items : 0;

    constexpr int Q = R::CHUNK / 4, RSTEP = 32 / Q;
    const int q = lane % Q, r0 = lane / Q;
    struct Place { int item, span, k; };                                     // of the next chunk to load, counted on without divisions
    Place pw = {(int)blockIdx.x, first, 0}, pa = pw;
    auto next = [&](Place& p) {
        p.k += R::CHUNK;
        if (p.k == parts(p.span) * R::CHUNK) {
            p.k = 0;
            p.span += wb;
            if (p.span >= spans) { p.span = first; p.item += gridDim.x; }
        }
    };
    auto load_w = [&](int slot) {
        float* st = ring + slot * R::STAGE + r0 * R::PAD + 4 * q;
        const int n0 = pw.item * rows_item + my_row, kb = pw.span * GR_SPAN + pw.k + 4 * q;
#pragma unroll
        for (int i = 0; i < GR_LANES * GR_ROWS / RSTEP; ++i) {
            const int lr = r0 + RSTEP * i, n = n0 + lr % GR_ROWS, k = kb + lr / GR_ROWS * BLOCK;
            const bool ok = n < N && k < K;
            cp_async<16>(st + RSTEP * i * R::PAD, ok ? W + (size_t)n * ldw + k : W, ok);
        }
        next(pw);
    };
    auto load_a = [&](int slot) {
        float* st = ring + slot * R::STAGE + R::W_FLOATS + r0 * R::PAD + 4 * q;
        const int kb = pa.span * GR_SPAN + pa.k + 4 * q;
#pragma unroll
        for (int i = 0; i < (GR_LANES * MT + RSTEP - 1) / RSTEP; ++i) {
            const int lm = r0 + RSTEP * i, m = m0 + lm % MT, k = kb + lm / MT * BLOCK;
            const bool ok = m < M && k < K;
            if (GR_LANES * MT % RSTEP == 0 || lm < GR_LANES * MT) cp_async<16>(st + RSTEP * i * R::PAD, ok ? A + (size_t)m * lda + k : A, ok);
        }
        next(pa);
    };
    // the weights of the first chunks are nobody's output: they are requested before the kernel ahead has finished
#pragma unroll
    for (int c = 0; c < GR_STAGES - 1; ++c)
        if (c < chunks) load_w(c);
    pdl_wait();
#pragma unroll
    for (int c = 0; c < GR_STAGES - 1; ++c) {
        if (c < chunks) load_a(c);
        cp_commit();
    }

    const int row = lane % GR_ROWS, blk = lane / GR_ROWS;
    int c = 0, slot = 0;
    for (int i = 0; i < n_items; ++i) {
        float* sum = sums + (i & 1) * sums_floats;
        for (int sp = 0; sp < mine; ++sp) {
            float acc[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[m] = 0.f;
            for (int part = parts(first + sp * wb); part > 0; --part, ++c) {
                if (c + GR_STAGES - 1 < chunks) {
                    const int to = slot == 0 ? GR_STAGES - 1 : slot - 1;
                    load_w(to);
                    load_a(to);
                }
                cp_commit();
                cp_wait<GR_STAGES - 1>();
                __syncwarp();
                const float* w = ring + slot * R::STAGE + lane * R::PAD;     // block * 8 + row
                const float* a = ring + slot * R::STAGE + R::W_FLOATS + blk * MT * R::PAD;
#pragma unroll 8
                for (int k = 0; k < R::CHUNK; k += 4) {
                    const float4 wv = *reinterpret_cast<const float4*>(w + k);
                    float4 av[MT];
#pragma unroll
                    for (int m = 0; m < MT; ++m) av[m] = *reinterpret_cast<const float4*>(a + m * R::PAD + k);
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[m] = fmaf(av[m].x, wv.x, acc[m]);
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[m] = fmaf(av[m].y, wv.y, acc[m]);
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[m] = fmaf(av[m].z, wv.z, acc[m]);
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[m] = fmaf(av[m].w, wv.w, acc[m]);
                }
                __syncwarp();                                    // the chunk is read before its place is filled again
                slot = slot == GR_STAGES - 1 ? 0 : slot + 1;
            }
            const int b = (first + sp * wb) * GR_LANES + blk;
#pragma unroll
            for (int m = 0; m < MT; ++m) sum[(b * MT + m) * rows_item + my_row + row] = acc[m];
        }
        __syncthreads();                                         // two sets of sums: the next item writes the other one
        for (int e = threadIdx.x; e < MT * rows_item; e += GR_WARPS * 32) {
            const int n = (blockIdx.x + i * gridDim.x) * rows_item + e % rows_item, m = m0 + e / rows_item;
            if (n >= N || m >= M) continue;
            float s = sum[e];
            for (int b = 1; b < nb; ++b) s += sum[b * MT * rows_item + e];
            C[(size_t)m * ldc + n] = s;
        }
    }
}

// ------------------------------------------------------------------------------------------------ tiles

constexpr int GT_THREADS = 128, GT_BK = 16;

// Threads TX x TY = 128 with TM x TN outputs each (TM a multiple of four): the tile is (TM * TY) x (TN * TX).  The small tile is for few
// CTAs, where a step waits for memory: its ring holds seven steps ahead (49 KB) instead of two.
template <int TM, int TN, int TX>
struct Tile {
    static constexpr int STAGES = TM * TN < 64 ? 8 : 3;
    static constexpr int TY = GT_THREADS / TX, BM = TM * TY, BN = TN * TX;
    static constexpr int A_ROW = BM + 4, W_ROW = GT_BK + 4;      // floats of a k of A and of a row of W: no two lanes of a phase on one bank
    static constexpr int A_FLOATS = GT_BK * A_ROW, STAGE = A_FLOATS + BN * W_ROW;
    static constexpr int SLOT = TM * TN * GT_THREADS;            // the outputs' sums, [output][thread]
};

// `ranks` CTAs of a cluster share a tile: rank r takes blocks r * per .. of K and keeps the sum of each in a slot of its own.  ranks = 1:
// one CTA takes all of them and one slot holds the running sum.
template <typename TI, typename TO, bool VEC, int TM, int TN, int TX>
__global__ void __launch_bounds__(GT_THREADS, 3)
gemm_tile_kernel(const TI* __restrict__ A, int lda, const TI* __restrict__ W, int ldw, TO* __restrict__ C, int ldc,
                 int M, int N, int K, int ranks, int per) {
    using T = Tile<TM, TN, TX>;
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float gt_smem[];
    float* slots = gt_smem + T::STAGES * T::STAGE;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a warp is 8 columns by 4 rows of threads
    const int tx = (warp % (TX / 8)) * 8 + lane % 8, ty = (warp / (TX / 8)) * 4 + lane / 8;
    const int rank = blockIdx.x % ranks;
    const int n0 = (blockIdx.x / ranks) * T::BN, m0 = blockIdx.y * T::BM;
    const int k_lo = rank * per * BLOCK, k_hi = min(K, (rank + 1) * per * BLOCK);
    const int steps = k_hi > k_lo ? (k_hi - k_lo + GT_BK - 1) / GT_BK : 0;

    static_assert(T::BN * GT_BK % (4 * GT_THREADS) == 0 && T::BM * GT_BK % GT_THREADS == 0, "whole rounds of copies");
    auto load = [&](int s) {                                     // VEC: a step's copies on their way
        float* sa = gt_smem + (s % T::STAGES) * T::STAGE;
        float* sw = sa + T::A_FLOATS;
        const int kb = k_lo + s * GT_BK;
        constexpr int COPIES = T::BN * (GT_BK / 4);
#pragma unroll
        for (int i = 0; i < COPIES / GT_THREADS; ++i) {
            const int e = tid + GT_THREADS * i, q = e % (GT_BK / 4), r = e / (GT_BK / 4), k = kb + 4 * q;
            const bool ok = n0 + r < N && k < k_hi;
            cp_async<16>(sw + r * T::W_ROW + 4 * q, ok ? W + (size_t)(n0 + r) * ldw + k : W, ok);
        }
        // a warp copies 8 k (a sector) of four rows: 32 banks of A's transposed place
#pragma unroll
        for (int i = 0; i < T::BM * GT_BK / GT_THREADS; ++i) {
            const int e = tid + GT_THREADS * i, r = e % 4 + e / 32 % (T::BM / 4) * 4, q = e / 4 % 8 + e / (8 * T::BM) * 8, k = kb + q;
            const bool ok = m0 + r < M && k < k_hi;
            cp_async<4>(sa + q * T::A_ROW + r, ok ? A + (size_t)(m0 + r) * lda + k : A, ok);
        }
    };
    // Else (bfloat16, or rows on no 16-byte boundary) GROUP steps are fetched into registers while the GROUP before is worked, and laid
    // down behind it: 64 x 64 x 172 of bfloat16 8.4 us, 18.2 when every step
    // waited for its own elements.
    constexpr int GROUP = VEC ? 1 : T::STAGES >= 8 ? 4 : 1, WE = VEC ? 1 : T::BN * GT_BK / GT_THREADS, AE = VEC ? 1 : T::BM * GT_BK / GT_THREADS;
    static_assert(VEC || T::STAGES >= 2 * GROUP, "the group that is worked and the next one");
    TI rw[GROUP][WE], ra[GROUP][AE];
    auto fetch = [&](int s0) {
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
            const int kb = k_lo + (s0 + u) * GT_BK;
#pragma unroll
            for (int i = 0; i < WE; ++i) {
                const int e = tid + GT_THREADS * i, q = e % GT_BK, r = e / GT_BK;
                rw[u][i] = n0 + r < N && kb + q < k_hi ? W[(size_t)(n0 + r) * ldw + kb + q] : from_f32<TI>(0.f);
            }
#pragma unroll
            for (int i = 0; i < AE; ++i) {
                const int e = tid + GT_THREADS * i, q = e % GT_BK, r = e / GT_BK;
                ra[u][i] = m0 + r < M && kb + q < k_hi ? A[(size_t)(m0 + r) * lda + kb + q] : from_f32<TI>(0.f);
            }
        }
    };
    auto lay = [&](int s0) {
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
            float* sa = gt_smem + ((s0 + u) % T::STAGES) * T::STAGE;
            float* sw = sa + T::A_FLOATS;
#pragma unroll
            for (int i = 0; i < WE; ++i) {
                const int e = tid + GT_THREADS * i;
                sw[e / GT_BK * T::W_ROW + e % GT_BK] = to_f32(rw[u][i]);
            }
#pragma unroll
            for (int i = 0; i < AE; ++i) {
                const int e = tid + GT_THREADS * i;
                sa[e % GT_BK * T::A_ROW + e / GT_BK] = to_f32(ra[u][i]);
            }
        }
    };

    f32x2 acc[TM / 2][TN];                                       // rows 4 * ty + (0, 1), (2, 3), then 4 * TY further on
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0;
    auto work = [&](int s) {
        const float* as = gt_smem + (s % T::STAGES) * T::STAGE + ty * 4;
        const float* ws = gt_smem + (s % T::STAGES) * T::STAGE + T::A_FLOATS + tx * T::W_ROW;
#pragma unroll
        for (int k = 0; k < GT_BK; k += 4) {
            float4 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + j * TX * T::W_ROW + k);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                f32x2 a[TM / 2];
#pragma unroll
                for (int i = 0; i < TM / 4; ++i) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(as + (k + kk) * T::A_ROW + i * 4 * T::TY);
                    a[2 * i] = v.x;
                    a[2 * i + 1] = v.y;
                }
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float wv = kk == 0 ? w[j].x : kk == 1 ? w[j].y : kk == 2 ? w[j].z : w[j].w;
                    const f32x2 ww = pair(wv, wv);
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i) acc[i][j] = fma2(a[i], ww, acc[i][j]);
                }
            }
        }
        constexpr int BLOCK_STEPS = BLOCK / GT_BK;
        if ((s + 1) % BLOCK_STEPS == 0 || s + 1 == steps) {      // a block is done
            const int b = s / BLOCK_STEPS;
            float* slot = slots + (ranks > 1 ? b * T::SLOT : 0) + tid;
            const bool add = ranks == 1 && b > 0;
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float2 v = unpair(acc[i][j]);
                    float *p = slot + (2 * i * TN + j) * GT_THREADS, *p2 = p + TN * GT_THREADS;
                    *p = add ? *p + v.x : v.x;
                    *p2 = add ? *p2 + v.y : v.y;
                    acc[i][j] = 0;
                }
        }
    };
    if constexpr (VEC) {
#pragma unroll
        for (int s = 0; s < T::STAGES - 1; ++s) {
            if (s < steps) load(s);
            cp_commit();
        }
        for (int s = 0; s < steps; ++s) {
            cp_wait<T::STAGES - 2>();
            __syncthreads();                                     // step s is here, and everyone has read step s - 1
            if (s + T::STAGES - 1 < steps) load(s + T::STAGES - 1);
            cp_commit();
            work(s);
        }
    } else if (steps > 0) {
        fetch(0);
        lay(0);
        for (int s0 = 0; s0 < steps; s0 += GROUP) {
            __syncthreads();                                     // this group is here, and everyone has read the one before
            const bool more = s0 + GROUP < steps;
            if (more) fetch(s0 + GROUP);
#pragma unroll 1
            for (int s = s0; s < min(s0 + GROUP, steps); ++s) work(s);
            if (more) lay(s0 + GROUP);
        }
    }

    auto store = [&](int e, float v) {
        const int i = e / TN;
        const int gm = m0 + i / 4 * 4 * T::TY + 4 * ty + i % 4, gn = n0 + tx + e % TN * TX;
        if (gm < M && gn < N) C[(size_t)gm * ldc + gn] = from_f32<TO>(v);
    };
    if (ranks == 1) {                                            // a thread reads what it wrote itself
#pragma unroll 4
        for (int e = 0; e < TM * TN; ++e) store(e, slots[e * GT_THREADS + tid]);
        return;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int nb = (K + BLOCK - 1) / BLOCK;
    const int e_lo = rank * TM * TN / ranks, e_hi = (rank + 1) * TM * TN / ranks;
    for (int e = e_lo; e < e_hi; ++e) {
        float s = 0.f;
        for (int b = 0; b < nb; ++b) {
            const float v = *cluster.map_shared_rank(slots + (b % per) * T::SLOT + e * GT_THREADS + tid, b / per);
            s = b == 0 ? v : s + v;
        }
        store(e, s);
    }
    cluster.sync();                                              // nobody leaves while its sums are read
}

template <typename TI, typename TO, bool VEC, int TM, int TN, int TX>
int launch_tiles(const TI* A, int lda, const TI* W, int ldw, TO* C, int ldc, int M, int N, int K, int ranks, cudaStream_t stream) {
    using T = Tile<TM, TN, TX>;
    const int nb = (K + BLOCK - 1) / BLOCK, per = (nb + ranks - 1) / ranks;
    const dim3 grid((N + T::BN - 1) / T::BN * ranks, (M + T::BM - 1) / T::BM);
    if (grid.y > 65535) return KL_ERR_BAD_SIZE;
    const size_t smem = (size_t)(T::STAGES * T::STAGE + (ranks > 1 ? per : 1) * T::SLOT) * sizeof(float);
    auto kernel = gemm_tile_kernel<TI, TO, VEC, TM, TN, TX>;
    KL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_kernel_clustered(kernel, ranks, grid, dim3(GT_THREADS), smem, stream, A, lda, W, ldw, C, ldc, M, N, K, ranks, per);
    return KL_OK;
}

template <typename TI, typename TO, bool VEC>
int tiles(const TI* A, int lda, const TI* W, int ldw, TO* C, int ldc, int M, int N, int K, cudaStream_t stream) {
    using Big = Tile<8, 8, 16>;
    const int sms = sm_count() > 0 ? sm_count() : 1, nb = (K + BLOCK - 1) / BLOCK;
    const long long big = (long long)((N + Big::BN - 1) / Big::BN) * ((M + Big::BM - 1) / Big::BM);
    // Where the tiles do not fill the device four times, the blocks of K are dealt to a cluster (at most two a CTA: a block's sums take 32 KB).
    // Where they do, a CTA keeps one running sum (77 KB, three CTAs an SM instead of two, and no sums to exchange): us with a cluster / without,
    // 777 x 16,384 x 2,048 1,367 / 1,257, 777 x 28,672 x 4,096 4,759 / 4,117, 777 x 9,000 x 1,100 804 / 410.
    int ranks = 1;
    if (nb <= 16 && big < 4LL * sms)
        while (ranks < 8 && ranks < nb && (big * ranks < 4LL * sms || (nb + ranks - 1) / ranks > 2)) ranks *= 2;
    if (ranks > 1 && (nb + ranks - 1) / ranks > 2) ranks = 1;
    if (2 * big * ranks >= 3LL * sms)
        return launch_tiles<TI, TO, VEC, 8, 8, 16>(A, lda, W, ldw, C, ldc, M, N, K, ranks, stream);
    return launch_tiles<TI, TO, VEC, 4, 4, 8>(A, lda, W, ldw, C, ldc, M, N, K, ranks, stream);
}

template <int MT>
int rows(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, cudaStream_t stream) {
    using R = Rows<MT>;
    const int nb = (K + BLOCK - 1) / BLOCK, spans = (nb + GR_LANES - 1) / GR_LANES;
    const int wb = spans >= 4 ? 4 : spans >= 2 ? 2 : 1, rows_item = GR_ROWS * (GR_WARPS / wb), items = (N + rows_item - 1) / rows_item;
    const size_t smem = (size_t)(GR_WARPS * GR_STAGES * R::STAGE + 2 * spans * GR_LANES * MT * rows_item) * sizeof(float);
    const auto kernel = K - (spans - 1) * GR_SPAN > BLOCK - R::CHUNK ? gemm_rows_kernel<MT, true> : gemm_rows_kernel<MT, false>;
    KL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // Two CTAs an SM, although shared memory holds one (118 KB for one row; two for three and four rows): the second ones start where the
    // first ones end.  us with this grid / with one CTA an SM, one row: 16,384 x 2,048 30.2 / 32.0, 32,000 x 2,048 59.5 / 59.5, 4,096 x 4,096
    // 16.3 / 15.7, 2,048 x 8,192 15.0 / 13.5; eight rows: 64.2 / 66.1, 2,048 x 8,192 33.1 / 29.9.
    const int most = 2 * (sm_count() > 0 ? sm_count() : 1);
    launch_kernel(kernel, dim3(items < most ? items : most, (M + MT - 1) / MT), dim3(GR_WARPS * 32), smem, stream, A, lda, W, ldw,
                  C, ldc, M, N, K, wb);
    return KL_OK;
}

// Up to 16 rows read W again for every 8 (16 rows, N = 2,048, K = 2,048 / N = 16,384: 18 / 122 us; the tiles take 35 / 123 for 33 rows);
// 24 rows would take 34 / 186.  The sums of up to 128 blocks of K fit beside the ring.
constexpr int ROWS_MAX_M = 16, ROWS_MAX_K = 65536;

}  // namespace kl

using namespace kl;

// in_dtype: dtype of A and W; out_dtype: dtype of C (float32 output of bfloat16 operands is
// what the classifier uses for logits).
KL_API int kl_gemm_simt(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N, int K,
                        int in_dtype, int out_dtype, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return KL_OK;
    if (K <= 0) return KL_ERR_BAD_SIZE;
    int err = KL_OK;
    if (in_dtype == KL_F32 && out_dtype == KL_F32) {
        const float *a = (const float*)A, *w = (const float*)W;
        float* c = (float*)C;
        // 16-byte copies need rows of whole 16-byte pieces on 16-byte boundaries
        const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) % 16 == 0;
        if (vec && M <= ROWS_MAX_M && K <= ROWS_MAX_K) {
            err = M == 1 ? rows<1>(a, lda, w, ldw, c, ldc, M, N, K, stream) : M == 2 ? rows<2>(a, lda, w, ldw, c, ldc, M, N, K, stream)
                : M <= 4 ? rows<4>(a, lda, w, ldw, c, ldc, M, N, K, stream) : rows<8>(a, lda, w, ldw, c, ldc, M, N, K, stream);
        } else if (vec) {
            err = tiles<float, float, true>(a, lda, w, ldw, c, ldc, M, N, K, stream);
        } else {
            err = tiles<float, float, false>(a, lda, w, ldw, c, ldc, M, N, K, stream);
        }
    } else if (in_dtype == KL_BF16 && out_dtype == KL_BF16) {
        err = tiles<bf16, bf16, false>((const bf16*)A, lda, (const bf16*)W, ldw, (bf16*)C, ldc, M, N, K, stream);
    } else if (in_dtype == KL_BF16 && out_dtype == KL_F32) {
        err = tiles<bf16, float, false>((const bf16*)A, lda, (const bf16*)W, ldw, (float*)C, ldc, M, N, K, stream);
    } else {
        return KL_ERR_BAD_DTYPE;
    }
    if (err != KL_OK) return err;
    KL_LAUNCH_CHECK();
    return KL_OK;
}
