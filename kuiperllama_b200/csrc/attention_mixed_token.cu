// The mixed-head attention of attention_mixed.cu for steps of single tokens over caches of bfloat16:
//
//   s_h(j) = scale * q_h . k_kv(h)(j);   s <- cap * tanh(s / cap);   s <- s - r1_h * ln(1 + r2_h * (i - j))
//   p_h = softmax over the visible keys;   w_h(j) = sum_g talk[h, g] p_g(j);   out_h = gate * sum_j w_h(j) v_kv(h)(j)
//
// One launch.  A cluster of up to eight CTAs has a sequence and all its heads; its visible chunks of 32 keys are dealt to the CTAs in turn.  A CTA
//
//   scores   reads its keys once: a warp takes 16 keys of a key/value head, mma.m16n8k16 with the head's queries as columns (exact products,
//            32-bit sums), and then the soft cap, the bias and the mask a key a lane.  All scores of the CTA stay in shared memory
//   softmax  takes them to exp(s - m) with its own maximum m, trades maxima and sums with the other CTAs through distributed shared memory, and
//            puts exp(m - M) / L of every head into the columns of talk
//   mix      W = talk P over the P that it has read, both as three bfloat16 numbers each (24 bits of mantissa, pieces.cuh)
//   values   O += W V: w as three bfloat16 numbers, the pieces of four heads as 12 rows of one tile.  A product starts from zero and is added with
//            rounding, the pieces meet at the end
//   out      adds the CTAs' pieces in their order, a part of the heads each
//
// One more warp fills a ring of slots by TMA, a whole chunk of all key/value heads a copy, the values' first chunks while the last scores are worked.
// Where a CTA has more chunks than its shared memory holds the scores of, they are worked in rounds and the scores computed twice.
// What bounds it is the latency of these steps (about 9 us for one chunk) and the instructions of a chunk, 1.1 us with 32 heads of 64 on 8: the caches of
// 64 sequences of 1,000 keys take 20 of its 45 us.  With 32 heads of 64 on 8, window 1,024 and 64 kept keys, us by attention_mixed_tiled.cu (a score computed
// twice, three barriers a chunk, 32-bit FMA through shared memory, pieces in a second and third launch) / here: 64 sequences of 200 keys 64.5 / 16.8, of 30
// 22.9 / 11.1, of 1,000 227 / 45; one of 1,000 32.2 / 17.2; 148 of 200 89 / 23; of 8,000 without a window 64 1,683 / 351, four 176 / 79.  Keys and values
// through cp.async by all threads took 22.5 for 64 of 200, one thread of the sixteen warps issuing TMA 18.2.
//
// ExiledOfCode/KuiperLLama's attention is mha_kernel.cu:61,74-106 (one sequence, one query, no window, no bias).
#include "common.cuh"
#include "pieces.cuh"
#include "soft_cap.cuh"
#include "tma_host.cuh"

namespace kl {

constexpr int MK_WARPS = 16, MK_THREADS = MK_WARPS * 32, MK_CH = 32;       // one more warp copies
constexpr int MK_HEADS = 64;                      // at most: four a warp in the softmax, four tiles of 16 rows of talk
constexpr int MK_SLOTS = 4;                       // at most
constexpr int MK_RANKS = 8;                       // CTAs of a cluster, at most

struct MixedTokenArgs {
    const bf16* q; long long q_stride;
    const bf16* gate; long long gate_stride;
    bf16* out; long long out_stride;
    const int* block_table; int blocks_per_seq;
    const int* cu_tokens; const int* seq_slots; const int* seq_starts;
    const float* r1; const float* r2; const float* talk;
    int* status;
    int heads, kv_heads, window, keep_first;
    int slots, room;                              // slots of the ring; chunks whose scores shared memory holds
    float scale, softcap, out_scale;
    float scale_cap, scale_cap_rest;              // scale / softcap as the sum of two numbers
};

// byte offsets in shared memory
struct MixedTokenLayout {
    uint32_t scores, rest, talk, ml, fac, q, bars, total;
    int J, Hp, share;                             // floats of a head's scores; heads as whole tiles of 16; heads whose sums a CTA adds
    __host__ __device__ MixedTokenLayout(int H, int G, int D, int slots, int room, bool mix, int ranks) {
        J = room * MK_CH + 8;
        Hp = (H + 15) & ~15;
        share = (H + ranks - 1) / ranks;
        scores = (uint32_t)slots * G * MK_CH * D * 2;                      // the ring [slots][G][32][D] before them; [H][J]
        rest = scores + (uint32_t)H * J * 4;                               // [ranks][share][D]: every CTA's sums of this CTA's heads
        talk = rest + (uint32_t)ranks * share * D * 4;                     // [3][Hp][Hp + 8]: talk in three pieces
        ml = talk + (mix ? (uint32_t)3 * Hp * (Hp + 8) * 2 : 0);           // [ranks][H]: every CTA's maxima and sums
        fac = ml + (uint32_t)ranks * Hp * 8;                               // [H]
        q = fac + (uint32_t)Hp * 4;                                        // [H][D + 8]
        bars = q + (uint32_t)Hp * (D + 8) * 2;
        total = bars + 2 * MK_SLOTS * 8 + 16;
    }
};

// where 16-byte piece c of a key's row lies in a tile of 32 rows of D elements as TMA's 128-byte swizzle leaves them (D = 32: two keys a line; D = 128:
// two boxes of 64 elements, `box` elements apart)
template <int D> __device__ __forceinline__ int mk_at(int r, int c, int box) {
    if constexpr (D == 32) return (r >> 1) * 64 + ((((r & 1) * 4 + c) ^ ((r >> 1) & 7)) << 3);
    else return (c >> 3) * box + r * 64 + (((c & 7) ^ (r & 7)) << 3);
}

__device__ __forceinline__ void mk_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void mk_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void mk_push(uint32_t addr, float a, float b) {       // to a shared::cluster address
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}

// UPW: (key/value head, four of its heads, 32 columns) pieces of O per warp, at most
template <int D, int UPW>
__global__ void __launch_bounds__(MK_THREADS + 32, 1)
attention_mixed_token_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const MixedTokenArgs A) {
    constexpr int W = D + 8, SL = D / 32;                                  // elements of a query's row; column slices
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(1024) unsigned char mk_raw[];
    const int ranks = gridDim.x, rank = ranks > 1 ? (int)cluster_ctarank() : 0;
    const int s = blockIdx.y, row = A.cu_tokens[s], row_end = A.cu_tokens[s + 1], i = A.seq_starts[s];
    const int* table = A.block_table + (size_t)A.seq_slots[s] * A.blocks_per_seq;
    if (row_end <= row) return;                                            // (the whole cluster)
    if (ranks > 1) mk_cluster_arrive();                                    // (this CTA runs: the others may write into its shared memory)
    const int H = A.heads, G = A.kv_heads, per = H / G, S = A.slots, room = A.room;
    const MixedTokenLayout L(H, G, D, S, room, A.talk != nullptr, ranks);
    const int J = L.J, Hp = L.Hp;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, t2 = (lane & 3) * 2;
    bf16* Ring = reinterpret_cast<bf16*>(mk_raw);
    float* Ps = reinterpret_cast<float*>(mk_raw + L.scores);
    float* rest = reinterpret_cast<float*>(mk_raw + L.rest);
    bf16* Ts = reinterpret_cast<bf16*>(mk_raw + L.talk);
    float* ml = reinterpret_cast<float*>(mk_raw + L.ml);
    float* fac = reinterpret_cast<float*>(mk_raw + L.fac);
    bf16* Qs = reinterpret_cast<bf16*>(mk_raw + L.q);
    uint64_t* full = reinterpret_cast<uint64_t*>(mk_raw + L.bars);
    uint64_t* empty = full + MK_SLOTS;
    volatile int* gave_up = reinterpret_cast<volatile int*>(empty + MK_SLOTS);
    const int slot = G * MK_CH * D, box = G * MK_CH * 64;                  // elements of a chunk, and of a box of 64 columns

    // chunks that neither the window nor the kept first keys reach are skipped; every `ranks`-th of the others is this CTA's
    const int chunks = i / MK_CH + 1;
    const int first = A.window > 0 ? max(0, i - A.window + 1) / MK_CH : 0;
    const int keep = A.window > 0 ? A.keep_first : 0;
    const int kept = min(first, (keep + MK_CH - 1) / MK_CH);
    const int visible = kept + chunks - first;
    const int n = rank < visible ? (visible - rank + ranks - 1) / ranks : 0;
    const int rounds = (n + room - 1) / room;
    auto chunk_of = [&](int t) {
        const int v = rank + t * ranks;
        return v < kept ? v : v - kept + first;
    };
    // the ring's items: the keys of all chunks, then each round's values (behind its keys once more where there are several rounds)
    const int items = n + (rounds > 1 ? 2 * n : n);
    auto item = [&](int x, bool& values) {
        values = false;
        if (x < n) return x;
        x -= n;
        values = true;
        if (rounds <= 1) return x;
        const int rd = x / (2 * room), o = x - rd * 2 * room, count = min(room, n - rd * room);
        values = o >= count;
        return rd * room + (values ? o - count : o);
    };
    if (threadIdx.x == 0) {
        for (int z = 0; z < S; ++z) { mbar_init(full + z, 1); mbar_init(empty + z, MK_WARPS); }
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == MK_WARPS) {                                                // ---- the copies: a slot is filled again when every warp has left it
        bool values;
        int page = items > 0 ? table[chunk_of(item(0, values)) * MK_CH / PAGE] : 0, at = 0, turn = 0, x = 0;
        auto fill = [&](int end) {
            for (; x < end; ++x) {
                const int t = item(x, values), y = chunk_of(t) * MK_CH % PAGE;
                bool later;
                const int page_next = x + 1 < items ? table[chunk_of(item(x + 1, later)) * MK_CH / PAGE] : 0;
                if (turn > 0 && !mbar_wait(empty + at, (turn - 1) & 1, gave_up, A.status, 23)) return;
                bf16* dst = Ring + (size_t)at * slot;
                mbar_expect_tx(full + at, (uint32_t)slot * 2);
                const CUtensorMap* map = values ? &map_v : &map_k;
                if constexpr (D == 32) tma_load_3d(dst, map, full + at, 0, y / 2, page * G);
                else
                    for (int c = 0; c < D / 64; ++c) tma_load_3d(dst + (size_t)c * box, map, full + at, c * 64, y, page * G);
                page = page_next;
                if (++at == S) { at = 0; ++turn; }
            }
        };
        // Its part in the cluster's three barriers: it reports to the second before it waits for a slot that is left only behind it
        if (lane == 0) fill(min(S, items));
        __syncwarp();
        if (ranks > 1) { mk_cluster_wait(); mk_cluster_arrive(); }
        if (lane == 0) fill(items);
        __syncwarp();
        if (ranks > 1) { mk_cluster_wait(); cluster_sync(); }
        return;
    }
    int at = 0, turn = 0;                                                  // the slot of the item in work
    auto here = [&]() {
        mbar_wait(full + at, turn & 1, gave_up, A.status, 24);
        return Ring + (size_t)at * slot;
    };
    auto done = [&]() {                                                    // this warp has left it
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + at);
        if (++at == S) { at = 0; ++turn; }
    };
    auto together = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(MK_THREADS) : "memory"); };

    for (int idx = threadIdx.x; idx < H * (W / 2); idx += MK_THREADS) {
        const int h = idx / (W / 2), e = (idx - h * (W / 2)) * 2;
        *reinterpret_cast<uint32_t*>(Qs + (size_t)h * W + e) =
            e < D ? *reinterpret_cast<const uint32_t*>(A.q + (size_t)row * A.q_stride + (size_t)h * D + e) : 0u;
    }
    float2 tk[MK_HEADS * MK_HEADS / 2 / MK_THREADS];                       // pairs of talk, rows and columns past the heads are zero
#pragma unroll
    for (int z = 0; z < MK_HEADS * MK_HEADS / 2 / MK_THREADS; ++z) {
        const int idx = threadIdx.x + z * MK_THREADS, h = idx / (Hp / 2), e = idx % (Hp / 2) * 2;
        tk[z] = make_float2(0.f, 0.f);
        if (A.talk != nullptr && h < H) {
            if (e < H) tk[z].x = A.talk[(size_t)h * H + e];
            if (e + 1 < H) tk[z].y = A.talk[(size_t)h * H + e + 1];
        }
    }
    float r1[4], r2[4], top[4], m[4], l[4];                                // of heads warp, warp + 16, ..
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int h = warp + u * MK_WARPS;
        r1[u] = A.r1 != nullptr && h < H ? A.r1[h] : 0.f;
        r2[u] = A.r1 != nullptr && h < H ? A.r2[h] : 0.f;
        m[u] = -INFINITY;
        l[u] = 0.f;
    }

    // ---- one chunk's products of queries and keys, into place o of the scores
    const int blocks8 = (per + 7) / 8;
    auto products = [&](const bf16* K, int o) {
        for (int unit = warp; unit < G * blocks8 * 2; unit += MK_WARPS) {
            const int half = unit & 1, g = (unit >> 1) / blocks8, h0 = ((unit >> 1) - g * blocks8) * 8;
            const bf16* k = K + (size_t)g * MK_CH * (D < 64 ? D : 64);
            const bf16* q = Qs + (size_t)(g * per + min(h0 + gid, per - 1)) * W + t2;
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                uint32_t a[4];
                pc_ldm4(smem_u32(k + mk_at<D>(half * 16 + (lane & 15), ks * 2 + (lane >> 4), box)), a);
                float more[4];                                             // (from zero and added with rounding: see pc_mma33)
                pc_mma0(more, a, *reinterpret_cast<const uint32_t*>(q + ks * 16), *reinterpret_cast<const uint32_t*>(q + ks * 16 + 8));
#pragma unroll
                for (int e = 0; e < 4; ++e) c[e] += more[e];
            }
            float* p = Ps + (size_t)(g * per + h0 + t2) * J + o * MK_CH + half * 16 + gid;
            if (h0 + t2 < per) { p[0] = c[0]; p[8] = c[2]; }
            if (h0 + t2 + 1 < per) { p[J] = c[1]; p[J + 8] = c[3]; }
        }
    };
    // ---- the soft cap, the bias and the mask of a chunk's scores: two heads per warp and turn, a key per lane
    auto finish = [&](int t, int o) {
        const int pos = chunk_of(t) * MK_CH + lane;
        const bool vis = pos <= i && (A.window == 0 || i - pos < A.window || pos < keep);
        const float away = (float)max(0, i - pos);
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
            const int h = warp + u * MK_WARPS;
            if (h >= H) break;
            const bool two = h + MK_WARPS < H;
            float* p = Ps + (size_t)h * J + o * MK_CH + lane;
            float* p2 = p + (two ? (size_t)MK_WARPS * J : 0);
            float v = *p, v2 = *p2;
            if (A.softcap > 0.f) {
                // (asked for every lane's own two scores: past the last key the page holds whatever was there before, and no visible score takes another
                // form for it)
                if (vis && fmaxf(fabsf(v), fabsf(v2)) * fabsf(A.scale_cap) > CAP_SMALL) {
                    v = tanhf(cap_quotient(v, A.scale_cap, A.scale_cap_rest));
                    v2 = tanhf(cap_quotient(v2, A.scale_cap, A.scale_cap_rest));
                } else {
                    v = cap_tanh(cap_small_quotient(v, A.scale_cap, A.scale_cap_rest));
                    v2 = cap_tanh(cap_small_quotient(v2, A.scale_cap, A.scale_cap_rest));
                }
            }
            const float factor = A.softcap > 0.f ? A.softcap : A.scale;
            if (A.r1 != nullptr) {
                v = fmaf(v, factor, -r1[u] * log1pf(r2[u] * away));
                v2 = fmaf(v2, factor, -r1[u + 1] * log1pf(r2[u + 1] * away));
            } else { v *= factor; v2 *= factor; }
            v = vis ? v : -INFINITY;
            v2 = vis ? v2 : -INFINITY;
            *p = v;
            top[u] = fmaxf(top[u], v);
            if (two) {
                *p2 = v2;
                top[u + 1] = fmaxf(top[u + 1], v2);
            }
        }
    };
    auto scores = [&](int t0, int count) {
#pragma unroll
        for (int u = 0; u < 4; ++u) top[u] = -INFINITY;
        together();                                                        // the queries are there; everybody is done with the weights in the scores' place
        for (int o = 0; o < count; ++o) {
            const bf16* K = here();
            products(K, o);
            done();
            if (o > 0) finish(t0 + o - 1, o - 1);                          // (whose products everybody has made)
            together();
        }
        finish(t0 + count - 1, count - 1);
    };
    // ---- exp(score - m) in place (0 where m = -inf: nothing is seen, or nothing but -inf); the sum of a lane's
    auto exponentials = [&](int u, int count) {
        const float at = m[u] == -INFINITY ? 0.f : m[u];
        float sum = 0.f;
        float* p = Ps + (size_t)(warp + u * MK_WARPS) * J + lane;
#pragma unroll 4
        for (int o = 0; o < count; ++o) {
            const float e = expf(p[o * MK_CH] - at);
            p[o * MK_CH] = e;
            sum += e;
        }
        return sum;
    };
    for (int rd = 0; rd < rounds; ++rd) {
        const int count = min(room, n - rd * room);
        scores(rd * room, count);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (warp + u * MK_WARPS >= H) break;
            const float before = m[u];
            m[u] = fmaxf(before, warp_max(top[u]));
            const float sum = warp_sum(exponentials(u, count));
            l[u] = (before == -INFINITY ? 0.f : l[u] * expf(before - m[u])) + sum;
        }
    }
    // ---- every CTA's maximum and sum to every CTA, and what this CTA's numbers are multiplied by
    if (ranks > 1) mk_cluster_wait();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int h = warp + u * MK_WARPS;
        if (h < H && lane < ranks) {
            float* to = ml + 2 * (rank * H + h);
            if (ranks > 1) mk_push(mapa(smem_u32(to), lane), m[u], l[u]);
            else { to[0] = m[u]; to[1] = l[u]; }
        }
    }
    if (ranks > 1) cluster_sync(); else together();
    if (threadIdx.x < H) {
        const int h = threadIdx.x;
        float all = -INFINITY, sum = 0.f;
        for (int z = 0; z < ranks; ++z) all = fmaxf(all, ml[2 * (z * H + h)]);
        for (int z = 0; z < ranks; ++z) {
            const float mz = ml[2 * (z * H + h)], lz = ml[2 * (z * H + h) + 1];
            if (lz > 0.f) sum += lz * expf(mz - all);
            else if (!(lz == 0.f)) sum = lz;                               // NaN stays
        }
        const float inverse = sum > 0.f ? 1.0f / sum : 0.f;
        // (every visible score -inf: no weights)
        fac[h] = all == -INFINITY ? __int_as_float(0x7fffffff) : expf(ml[2 * (rank * H + h)] - all) * inverse;
    }
    together();
    if (A.talk != nullptr)
#pragma unroll
        for (int z = 0; z < MK_HEADS * MK_HEADS / 2 / MK_THREADS; ++z) {
            const int idx = threadIdx.x + z * MK_THREADS, h = idx / (Hp / 2), e = idx % (Hp / 2) * 2;
            if (h >= Hp) break;
            uint32_t a, b, c;
            pc_split(tk[z].x * (e < H ? fac[e] : 0.f), tk[z].y * (e + 1 < H ? fac[e + 1] : 0.f), a, b, c);
            uint32_t* to = reinterpret_cast<uint32_t*>(Ts + (size_t)h * (Hp + 8) + e);
            to[0] = a;
            to[Hp * (Hp + 8) / 2] = b;
            to[Hp * (Hp + 8)] = c;
        }

    float O[UPW][4][4];
#pragma unroll
    for (int u = 0; u < UPW; ++u) pc_zero<4>(O[u]);
    const int blocks4 = (per + 3) / 4, pieces = G * blocks4 * SL;
    for (int rd = 0; rd < rounds; ++rd) {
        const int t0 = rd * room, count = min(room, n - t0);
        if (rounds > 1) {
            scores(t0, count);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (warp + u * MK_WARPS < H) exponentials(u, count);
        }
        together();
        if (A.talk != nullptr)                                             // eight keys a warp, all heads: W over the P that the warp has read
            for (int unit = warp; unit < count * (MK_CH / 8); unit += MK_WARPS) {
                float* p = Ps + unit * 8;
                float d[MK_HEADS / 16][1][4], e[MK_HEADS / 16][1][4];
#pragma unroll
                for (int z = 0; z < MK_HEADS / 16; ++z) { pc_zero<1>(d[z]); pc_zero<1>(e[z]); }
                for (int g0 = 0; g0 < Hp; g0 += 16) {
                    uint32_t b[3][1][2];
#pragma unroll
                    for (int z = 0; z < 2; ++z) {                          // (rows past the heads meet zeros of talk)
                        const float* pg = p + gid;
                        const int g = g0 + z * 8 + t2;
                        pc_split(pg[(size_t)min(g, H - 1) * J], pg[(size_t)min(g + 1, H - 1) * J], b[0][0][z], b[1][0][z], b[2][0][z]);
                    }
#pragma unroll
                    for (int z = 0; z < MK_HEADS / 16; ++z)
                        if (z * 16 < Hp) {
                            uint32_t a[3][4];
#pragma unroll
                            for (int y = 0; y < 3; ++y) pc_ldm4(smem_u32(Ts + (size_t)(y * Hp + z * 16 + (lane & 15)) * (Hp + 8) + g0 + (lane >> 4) * 8), a[y]);
                            float dd[1][4];
                            pc_mma33<1, false>(dd, e[z], a, b);
                            pc_add<1>(d[z], dd);
                        }
                }
                __syncwarp();
#pragma unroll
                for (int z = 0; z < MK_HEADS / 16; ++z)
                    if (z * 16 < Hp)
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const int h = z * 16 + gid + y * 8;
                            float2 w = make_float2(d[z][0][2 * y] + e[z][0][2 * y], d[z][0][2 * y + 1] + e[z][0][2 * y + 1]);
                            if (!(fabsf(w.x) < INFINITY)) w.x = d[z][0][2 * y];                 // (as for O below)
                            if (!(fabsf(w.y) < INFINITY)) w.y = d[z][0][2 * y + 1];
                            if (h < H) *reinterpret_cast<float2*>(p + (size_t)h * J + t2) = w;
                        }
            }
        together();                                                        // every chunk is mixed
        for (int o = 0; o < count; ++o) {
            bf16* V = here();
            const int live = i + 1 - chunk_of(t0 + o) * MK_CH;
            if (live < MK_CH) {                                            // rows past the last key: whatever the page holds there becomes zero
                for (int idx = threadIdx.x; idx < G * MK_CH * (D / 8); idx += MK_THREADS) {
                    const int r = idx / (D / 8) % MK_CH, g = idx / (D / 8) / MK_CH;
                    if (r >= live) *reinterpret_cast<uint4*>(V + (size_t)g * MK_CH * (D < 64 ? D : 64) + mk_at<D>(r, idx % (D / 8), box)) = make_uint4(0, 0, 0, 0);
                }
                together();
            }
#pragma unroll
            for (int u = 0; u < UPW; ++u) {
                const int unit = warp + u * MK_WARPS;
                if (unit >= pieces) break;
                const int sl = unit % SL, b = unit / SL, g = b / blocks4, h0 = (b - g * blocks4) * 4;
                const int h = g * per + min(h0 + (gid & 3), per - 1);
                const float* w = Ps + (size_t)h * J + o * MK_CH + t2;
                const float f = A.talk != nullptr ? 1.f : fac[h];
                float c[4][4];
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const float2 x0 = *reinterpret_cast<const float2*>(w + ks * 16), x1 = *reinterpret_cast<const float2*>(w + ks * 16 + 8);
                    uint32_t hi0, mid0, lo0, hi1, mid1, lo1;
                    pc_split(x0.x * f, x0.y * f, hi0, mid0, lo0);
                    pc_split(x1.x * f, x1.y * f, hi1, mid1, lo1);
                    // rows 0..3 the heads' leading pieces, 4..7 the middle ones, 8..11 the last
                    const uint32_t a[4] = {gid < 4 ? hi0 : mid0, gid < 4 ? lo0 : 0u, gid < 4 ? hi1 : mid1, gid < 4 ? lo1 : 0u};
                    const bf16* v = V + (size_t)g * MK_CH * (D < 64 ? D : 64);
#pragma unroll
                    for (int nt = 0; nt < 4; nt += 2) {
                        uint32_t bb[4];
                        pc_ldm4t(smem_u32(v + mk_at<D>(ks * 16 + (lane & 15), sl * 4 + nt + (lane >> 4), box)), bb);
                        if (ks == 0) { pc_mma0(c[nt], a, bb[0], bb[1]); pc_mma0(c[nt + 1], a, bb[2], bb[3]); }
                        else { pc_mma(c[nt], a, bb[0], bb[1]); pc_mma(c[nt + 1], a, bb[2], bb[3]); }
                    }
                }
                pc_add<4>(O[u], c);
            }
            done();
        }
    }
    // ---- the sums of every head to the CTA that adds them
#pragma unroll
    for (int u = 0; u < UPW; ++u) {
        const int unit = warp + u * MK_WARPS;
        if (unit >= pieces) break;
        const int sl = unit % SL, b = unit / SL, g = b / blocks4, h0 = (b - g * blocks4) * 4;
        const int h = g * per + h0 + (gid & 3), owner = h / L.share;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            float y[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float mid = __shfl_xor_sync(0xffffffffu, O[u][nt][e], 16);
                y[e] = O[u][nt][e] + (mid + O[u][nt][2 + e]);
                if (!(fabsf(y[e]) < INFINITY)) y[e] = O[u][nt][e];         // of an infinite number the leading piece is right, the others are NaN
            }
            if (gid < 4 && h0 + gid < per) {
                float* to = rest + (size_t)(rank * L.share + h - owner * L.share) * D + sl * 32 + nt * 8 + t2;
                if (ranks > 1) mk_push(mapa(smem_u32(to), owner), y[0], y[1]);
                else *reinterpret_cast<float2*>(to) = make_float2(y[0], y[1]);
            }
        }
    }
    if (ranks > 1) cluster_sync(); else together();
    const int h_first = rank * L.share, h_count = min(L.share, H - h_first);
    for (int idx = threadIdx.x * 2; idx < h_count * D; idx += MK_THREADS * 2) {
        float2 y = make_float2(0.f, 0.f);
        for (int z = 0; z < ranks; ++z) {
            const float2 v = *reinterpret_cast<const float2*>(rest + (size_t)z * L.share * D + idx);
            y.x += v.x; y.y += v.y;
        }
        const int h = h_first + idx / D;
        float f = A.out_scale;
        if (A.gate != nullptr) f *= 1.0f / (1.0f + expf(-to_f32(A.gate[(size_t)row * A.gate_stride + h])));
        *reinterpret_cast<__nv_bfloat162*>(A.out + (size_t)row * A.out_stride + (size_t)h_first * D + idx) = __floats2bfloat162_rn(y.x * f, y.y * f);
    }
}

struct MixedTokenPlan { int slots, room, upw; size_t smem; };
static MixedTokenPlan mixed_token_plan(int H, int G, int D, bool mix, int chunks, int ranks) {
    MixedTokenPlan P = {0, 0, 0, 0};
    if (H > MK_HEADS || (D != 32 && D != 64 && D != 128)) return P;
    const int units = G * ((H / G + 3) / 4) * (D / 32), upw = (units + MK_WARPS - 1) / MK_WARPS;
    if (upw > 4) return P;
    const long long most = 226 * 1024;
    auto bytes = [&](int slots, int room) {
        const MixedTokenLayout L(H, G, D, slots, room, mix, ranks);
        return (long long)L.total;
    };
    const long long a_chunk = (long long)H * MK_CH * 4;
    for (int slots = MK_SLOTS; slots >= 2; --slots)
        if (bytes(slots, 0) + chunks * a_chunk <= most) { P.slots = slots; P.room = chunks; break; }
    if (P.slots == 0) {                                                    // the scores in rounds
        const long long left = most - bytes(2, 0);
        if (left < 4 * a_chunk) return P;                                  // (fewer than four chunks at once: not here)
        P.slots = 2;
        P.room = (int)(left / a_chunk);
    }
    P.upw = upw <= 1 ? 1 : upw <= 2 ? 2 : 4;
    P.smem = (size_t)bytes(P.slots, P.room);
    return P;
}

static int mixed_token_map(CUtensorMap* map, const void* cache, int D, int G, long long pages) {
    // [pages * G][PAGE][D] in boxes of [G][32][64]; of 32 columns two keys are a row
    const int keys = D == 32 ? 2 : 1;
    const long long dims[3] = {(long long)D * keys, PAGE / keys, pages * G}, strides[2] = {(long long)D * keys, (long long)D * PAGE};
    const int box[3] = {64, MK_CH / keys, G};
    return tma_make_map(map, cache, 3, dims, strides, box);
}

}  // namespace kl

using namespace kl;

// 1 where kl_attention_mixed_token can run these sizes.
KL_API int kl_attention_mixed_token_fits(int heads, int kv_heads, int dim, int vdim, int has_talk) {
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || dim <= 0 || dim != vdim) return 0;
    return mixed_token_plan(heads, kv_heads, dim, has_talk != 0, 1 << 20, MK_RANKS).slots > 0;
}

// The chunks of 32 keys whose scores one of `ranks` CTAs keeps at once; of more it computes the scores twice, in rounds (0: sizes that do not run).
KL_API int kl_attention_mixed_token_room(int heads, int kv_heads, int dim, int has_talk, int ranks) {
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || dim <= 0 || ranks < 1 || ranks > MK_RANKS) return 0;
    return mixed_token_plan(heads, kv_heads, dim, has_talk != 0, 1 << 20, ranks).room;
}

// `ranks` (1, 2, 4 or 8) CTAs a sequence; `chunks`: the visible chunks of 32 keys that a CTA is planned for (more of them are right too, in rounds).
KL_API int kl_attention_mixed_token(const void* q, long long q_stride, const void* gate, long long gate_stride, void* out, long long out_stride,
                                    const void* k_cache, const void* v_cache, long long pages, const int* block_table, int blocks_per_seq,
                                    const int* cu_tokens, const int* seq_slots, const int* seq_starts, int n_seqs, int heads, int kv_heads, int dim,
                                    float scale, float softcap, const float* r1, const float* r2, const float* talk, int window, int keep_first,
                                    float out_scale, int ranks, int chunks, int* status, cudaStream_t stream) {
    if (n_seqs <= 0) return KL_OK;
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || window < 0 || keep_first < 0 || chunks < 1 || status == nullptr) return KL_ERR_BAD_SIZE;
    if ((ranks != 1 && ranks != 2 && ranks != 4 && ranks != 8) || (r1 == nullptr) != (r2 == nullptr) || n_seqs > 65535 || pages <= 0) return KL_ERR_BAD_SIZE;
    const MixedTokenPlan P = mixed_token_plan(heads, kv_heads, dim, talk != nullptr, chunks, ranks);
    if (P.slots == 0) return KL_ERR_BAD_SIZE;
    if ((((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) || (((uintptr_t)q | (uintptr_t)out) & 3) || ((q_stride | out_stride) & 1)) return KL_ERR_BAD_SIZE;
    CUtensorMap mk, mv;
    int rc = mixed_token_map(&mk, k_cache, dim, kv_heads, pages);
    if (rc == KL_OK) rc = mixed_token_map(&mv, v_cache, dim, kv_heads, pages);
    if (rc != KL_OK) return rc;
    MixedTokenArgs A;
    A.q = (const bf16*)q; A.q_stride = q_stride; A.gate = (const bf16*)gate; A.gate_stride = gate_stride; A.out = (bf16*)out; A.out_stride = out_stride;
    A.block_table = block_table; A.blocks_per_seq = blocks_per_seq;
    A.cu_tokens = cu_tokens; A.seq_slots = seq_slots; A.seq_starts = seq_starts; A.r1 = r1; A.r2 = r2; A.talk = talk; A.status = status;
    A.heads = heads; A.kv_heads = kv_heads; A.window = window; A.keep_first = keep_first; A.slots = P.slots; A.room = P.room;
    A.scale = scale; A.softcap = softcap; A.out_scale = out_scale;
    cap_parts(scale, softcap, A.scale_cap, A.scale_cap_rest);
#define KL_MK(DD, U)                                                                                                                          \
    do {                                                                                                                                      \
        KL_CUDA(cudaFuncSetAttribute(attention_mixed_token_kernel<DD, U>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem));         \
        launch_kernel_clustered(attention_mixed_token_kernel<DD, U>, ranks, dim3(ranks, n_seqs), dim3(MK_THREADS + 32), P.smem, stream, mk, mv, A); \
    } while (0)
#define KL_MK_BY_UPW(DD) do { if (P.upw == 1) KL_MK(DD, 1); else if (P.upw == 2) KL_MK(DD, 2); else KL_MK(DD, 4); } while (0)
    if (dim == 32) KL_MK_BY_UPW(32);
    else if (dim == 64) KL_MK_BY_UPW(64);
    else KL_MK_BY_UPW(128);
#undef KL_MK_BY_UPW
#undef KL_MK
    KL_LAUNCH_CHECK();
    return KL_OK;
}
