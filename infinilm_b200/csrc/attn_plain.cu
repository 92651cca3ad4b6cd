// Plain attention over the paged cache. It takes any mix of prompt portions and single decoded tokens, any head size up to
// 1024, any number of heads and groups, any page size and an optional window. It is the attention of the 32-bit path and the
// reference beside the fast bfloat16 kernels; all arithmetic is f32.
// With `sink` (one f32 number per query head) the softmax's denominator also holds exp(sink[head]): a key without a
// value whose score is the number itself, not multiplied by `scale`.
//
// The query of token t is at absolute position p = tok_pos[t] of its request and sees cache
// positions max(0, p - window + 1) .. p (window <= 0: all). Query head j reads kv head j / (nh / nkv).
// With `dist_bias` (f32 [dist_far + 1][heads]) the scaled score of a key n positions back gets dist_bias[min(n, dist_far)][head]
// added: a learned bias by distance that is constant from dist_far on.
// SIG: no softmax - a visible key's weight is the sigmoid of its (scaled, biased) score, and the weights are not
// normalised over the keys. CAP: the scaled score s becomes cap * tanh(s / cap) (a soft cap; the sink is not capped).
#include "common.cuh"

// ---- head sizes up to 256: tiles of 32 keys -----------------------------------------------------------------------------------
// A block serves one token and up to 8 query heads of one kv head (HW), a warp a head; with fewer heads, or few tokens in the
// step, several warps share a head and take tiles of 32 keys in turn (KS of them). A head's tiles go to R * KS running sums in turn,
// merged in their order at the end; how many there are follows from the heads alone, and whether two of them are two warps (R 1, few
// tokens) or one warp's in turn (R 2) from the tokens in the step. So a token's result is bit-identical whatever else is in the step. All warps of the block
// read the same keys and values from shared memory, where asynchronous copies bring the next round while this one is
// worked on (bfloat16, and sizes whose rows are not whole 16-byte pieces, are widened by plain loads instead). In the scores a lane
// is a key, in the weighted sum a pair of columns. What bounds it is the chain of a tile - scores, maximum, exponentials, sum -
// where one key at a time paid that chain and a trip to memory for every key: 16 heads on 2 of 64, one token over 80 keys 84 us, now 7.7; some 800 tokens of
// four prompts 1.3 ms, now 72 us.
constexpr int AT_KEYS = 32;
__host__ __device__ constexpr int at_row(int hdp) { return hdp + 4; }          // floats of a staged row: an odd number of 16-byte pieces
__host__ __device__ constexpr int at_round_floats(int hdp, int ks) { return 2 * ks * AT_KEYS * at_row(hdp); }

// What both kernels of these sizes do with a tile's scores, its weights and the running sums: one text, and the roundings spelled out, so that a
// token has the same bits from either.
// A lane's key: its score from the dot product's two halves, the sum's new maximum, the weight. `bias`: the key's, or null.
template <bool SIG, bool CAP, int NV>
__device__ __forceinline__ float at_weight(float d0, float d1, bool in, float scale, float cap, const float* bias, float& m, float& l, il_f2 (&acc)[NV]) {
    float s = __fmul_rn(__fadd_rn(d0, d1), scale);
    if (CAP) s = __fmul_rn(cap, tanhf(__fdiv_rn(s, cap)));
    if (bias) s = __fadd_rn(s, *bias);
    if constexpr (SIG) return in ? __fdiv_rn(1.f, __fadd_rn(1.f, expf(-s))) : 0.f;
    const float mn = fmaxf(m, il_warp_max(in ? s : -INFINITY));
    // exp(-inf) = 0 on the first tile; a tile whose scores are all -inf (a bias that masks) leaves the sum as it is
    const float ref = mn == -INFINITY ? 0.f : mn;
    const float corr = mn == -INFINITY ? 1.f : expf(__fadd_rn(m, -mn));
    const float p = in ? expf(__fadd_rn(s, -ref)) : 0.f;
    l = __fmaf_rn(l, corr, p);
    m = mn;
    const il_f2 c2 = il_f2_dup(corr);
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = il_f2_mul(acc[v], c2);
    return p;
}
// The first of a head's sums brought to the maximum m of all of them; then each other one's factor.
template <bool SIG, int NV> __device__ __forceinline__ void at_first(float m0, float m, float& l, il_f2 (&acc)[NV]) {
    if (SIG) return;
    const float c = m0 == -INFINITY ? 0.f : expf(__fadd_rn(m0, -m));
    l = __fmul_rn(l, c);
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = il_f2_mul(acc[v], il_f2_dup(c));
}
template <bool SIG> __device__ __forceinline__ float at_factor(float mi, float m) { return SIG ? 1.f : mi == -INFINITY ? 0.f : expf(__fadd_rn(mi, -m)); }
template <typename TA, bool SIG, int NV>
__device__ __forceinline__ void at_store(TA* orow, int hd, int lane, const float* sink, float m, float l, const il_f2 (&acc)[NV]) {
    if (sink) l = __fadd_rn(l, expf(__fadd_rn(*sink, -m)));      // (+inf when the sink towers over every score: the row is then zero)
    const float inv = SIG ? 1.f : __fdiv_rn(1.f, l);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        float a, b;
        il_f2_get(acc[v], a, b);
        const int d = 2 * lane + 64 * v;
        if (d < hd) orow[d] = il_from_f<TA>(__fmul_rn(a, inv));
        if (d + 1 < hd) orow[d + 1] = il_from_f<TA>(__fmul_rn(b, inv));
    }
}

template <typename TA, int HDP, bool SIG, bool CAP, int R>
__global__ void __launch_bounds__(R == 1 ? 512 : 256, R == 1 ? 2 : 4) attn_tile_kernel(const TA* qkv, int row_stride, TA* __restrict__ out, const TA* cache, const int* __restrict__ block_table,
                                 int bt_stride, const int* __restrict__ tok_pos, const int* __restrict__ tok_entry, int page_size, int page_shift,
                                 int nh, int nkv, int hd, float scale, int window, const float* __restrict__ sink,
                                 const float* __restrict__ dist_bias, int dist_far, float cap, int HW, int KS, int async) {
    extern __shared__ __align__(16) float sm[];
    il_pdl_wait();
    il_pdl_launch_dependents();                   // (a product behind may ask for its weights meanwhile)
    constexpr int RS = at_row(HDP), PIECES = HDP / 4, NV = (HDP + 63) / 64;
    const int G = nh / nkv, n_hb = (G + HW - 1) / HW;
    const int t = blockIdx.x, g = blockIdx.y / n_hb, hb = blockIdx.y - g * n_hb;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n_thr = blockDim.x;
    const int hs = warp % HW, ks = warp / HW;
    const int hj = hb * HW + hs;                  // head within the group
    const bool live = hj < G;
    const int j = g * G + (live ? hj : 0);
    const int round_f = at_round_floats(HDP, KS), half_f = KS * AT_KEYS * RS;
    float* qs = sm + 2 * round_f + (size_t)hs * HDP;             // this head's query
    float* ps = sm + 2 * round_f + HW * HDP + warp * AT_KEYS;    // this warp's weights of a tile
    const int pos = tok_pos[t];
    const int* bt = block_table + (size_t)tok_entry[t] * bt_stride;
    const int lo = il_mask_lo(pos, window), n_keys = pos - lo + 1;
    const int per_round = KS * AT_KEYS, rounds = (n_keys + per_round - 1) / per_round;
    const size_t page_elems = (size_t)2 * nkv * page_size * hd, v_off = (size_t)nkv * page_size * hd;
    auto load = [&](int r) {                      // keys lo + r * per_round ..: K rows, then V rows; rows past the last key are zero
        float* dst0 = sm + (r & 1) * round_f;
        for (int i = tid; i < per_round * PIECES; i += n_thr) {
            const int row = i / PIECES, d = (i % PIECES) * 4, kk = r * per_round + row;
            const bool in = kk < n_keys && d < hd;
            const int kp = lo + (kk < n_keys ? kk : 0);
            const int pi = page_shift >= 0 ? kp >> page_shift : kp / page_size;
            const TA* src = cache + (size_t)bt[pi] * page_elems + ((size_t)g * page_size + (kp - pi * page_size)) * hd + (d < hd ? d : 0);
            float* dst = dst0 + row * RS + d;
            if (sizeof(TA) == 4 && async) {
                const int bytes = in ? 16 : 0;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst + half_f)), "l"(src + v_off), "r"(bytes));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const bool ok = in && d + e < hd;
                    dst[e] = ok ? il_to_f(src[e]) : 0.f;
                    dst[half_f + e] = ok ? il_to_f(src[v_off + e]) : 0.f;
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    load(0);
    const TA* qrow = qkv + (size_t)t * row_stride + (size_t)j * hd;
    if (ks == 0)
        for (int d = lane; d < HDP; d += 32) qs[d] = d < hd ? il_to_f(qrow[d]) : 0.f;
    float m[R], l[R];                             // of the warp's sums; l: this lane's keys only
    il_f2 acc[R][NV];
#pragma unroll
    for (int u = 0; u < R; ++u) {
        m[u] = -INFINITY, l[u] = 0.f;
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[u][v] = 0ull;
    }
    for (int r0 = 0; r0 < rounds; r0 += R) {
#pragma unroll
        for (int u = 0; u < R; ++u) {             // round r goes to sum r % R: tile t of the keys to running sum t % (R * KS)
            const int r = r0 + u;
            if (R > 1 && r >= rounds) break;
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();                      // the round is there, and nobody reads the other half any more
            if (r + 1 < rounds) load(r + 1);
            const float* kr = sm + (r & 1) * round_f + (ks * AT_KEYS + lane) * RS;
            const int kk = r * per_round + ks * AT_KEYS + lane;
            const bool in = kk < n_keys;
            if (r * per_round + ks * AT_KEYS >= n_keys) continue;        // (warp-uniform: a tile without keys)
            il_f2 s2[2] = {0ull, 0ull};
#pragma unroll 8
            for (int d = 0; d < HDP; d += 4) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(kr + d), b = *reinterpret_cast<const ulonglong2*>(qs + d);
                s2[0] = il_f2_fma(a.x, b.x, s2[0]);
                s2[1] = il_f2_fma(a.y, b.y, s2[1]);
            }
            float d0, d1;
            il_f2_get(il_f2_add(s2[0], s2[1]), d0, d1);
            const float* bias = dist_bias && in ? dist_bias + (size_t)min(n_keys - 1 - kk, dist_far) * nh + j : nullptr;
            const float p = at_weight<SIG, CAP, NV>(d0, d1, in, scale, cap, bias, m[u], l[u], acc[u]);
            ps[lane] = p;
            __syncwarp();
            const float* vr = sm + (r & 1) * round_f + half_f + ks * AT_KEYS * RS + 2 * lane;
#pragma unroll 2
            for (int key = 0; key < AT_KEYS; key += 4) {
                const float4 w = *reinterpret_cast<const float4*>(ps + key);
                const float wk[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        if (HDP >= 64 || 2 * lane < HDP)
                            acc[u][v] = il_f2_fma(il_f2_dup(wk[e]), *reinterpret_cast<const il_f2*>(vr + (key + e) * RS + 64 * v), acc[u][v]);
            }
            __syncwarp();                         // ps is written again in the next round
        }
    }
    if (!SIG)
#pragma unroll
        for (int u = 0; u < R; ++u) l[u] = il_warp_sum(l[u]);
    if (R * KS > 1) {                             // the sums of a head: maxima, sums and weighted sums through shared memory
        __syncthreads();
#pragma unroll
        for (int u = 0; u < R; ++u) {             // sum u * KS + ks
            float* part = sm + (size_t)(u * KS * HW + warp) * (HDP + 4);
            if (lane == 0) part[HDP] = m[u], part[HDP + 1] = l[u];
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (HDP >= 64 || 2 * lane < HDP) *reinterpret_cast<il_f2*>(part + 2 * lane + 64 * v) = acc[u][v];
        }
        __syncthreads();
        if (ks != 0) return;
        const float m0 = m[0];
        for (int i = 1; i < R * KS; ++i) m[0] = fmaxf(m[0], sm[(size_t)(i * HW + hs) * (HDP + 4) + HDP]);
        at_first<SIG, NV>(m0, m[0], l[0], acc[0]);
        for (int i = 1; i < R * KS; ++i) {
            const float* other = sm + (size_t)(i * HW + hs) * (HDP + 4);
            const float c = at_factor<SIG>(other[HDP], m[0]);
            l[0] = __fmaf_rn(c, other[HDP + 1], l[0]);
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (HDP >= 64 || 2 * lane < HDP)
                    acc[0][v] = il_f2_fma(il_f2_dup(c), *reinterpret_cast<const il_f2*>(other + 2 * lane + 64 * v), acc[0][v]);
        }
    }
    if (live) at_store<TA, SIG, NV>(out + (size_t)t * nh * hd + (size_t)j * hd, hd, lane, sink ? sink + j : nullptr, m[0], l[0], acc[0]);
}

// The same for many tokens of heads that share no keys, or few do: there a block of the kernel above is 1 to 4 warps and 140 KB of tiles, one block an
// SM, and keys staged for them alone. Here a warp has a (token, head), holds all its running sums (V) and reads keys and values from memory, through L1: in the
// scores eight columns of its key's row a lane and load, in the weighted sum whole rows. What bounds it is the lines that the loads of 32 rows touch in L1; the
// (token, head) pairs an SM holds cover each other's chains.
constexpr int AT_DIRECT_WARPS = 4;
// Four elements p[0 .. 3] of a row as two pairs, zeros from `left` on. VEC: left is a multiple of 4 and the row aligned to four elements.
__device__ __forceinline__ void at_load4(const float* p, int left, bool vec, il_f2& lo, il_f2& hi) {
    if (vec) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        lo = il_f2_make(x.x, x.y), hi = il_f2_make(x.z, x.w);
    } else {
        lo = il_f2_make(p[0], left > 1 ? p[1] : 0.f), hi = il_f2_make(left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
    }
}
__device__ __forceinline__ void at_load4(const __nv_bfloat16* p, int left, bool vec, il_f2& lo, il_f2& hi) {
    if (vec) {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
        lo = il_f2_make(a.x, a.y), hi = il_f2_make(b.x, b.y);
    } else {
        lo = il_f2_make(il_to_f(p[0]), left > 1 ? il_to_f(p[1]) : 0.f), hi = il_f2_make(left > 2 ? il_to_f(p[2]) : 0.f, left > 3 ? il_to_f(p[3]) : 0.f);
    }
}
// Eight elements as four pairs: one load of 32 (16) bytes, aligned to as many.
__device__ __forceinline__ void at_load8(const float* p, il_f2 (&a)[4]) {
    float x[8];
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]) : "l"(p));
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = il_f2_make(x[2 * i], x[2 * i + 1]);
}
__device__ __forceinline__ void at_load8(const __nv_bfloat16* p, il_f2 (&a)[4]) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
        a[i] = il_f2_make(x.x, x.y);
    }
}
__device__ __forceinline__ il_f2 at_load2(const float* p, int left, bool vec) {
    if (vec) {
        const float2 x = *reinterpret_cast<const float2*>(p);
        return il_f2_make(x.x, x.y);
    }
    return il_f2_make(p[0], left > 1 ? p[1] : 0.f);
}
__device__ __forceinline__ il_f2 at_load2(const __nv_bfloat16* p, int left, bool vec) {
    if (vec) {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
        return il_f2_make(x.x, x.y);
    }
    return il_f2_make(il_to_f(p[0]), left > 1 ? il_to_f(p[1]) : 0.f);
}

template <typename TA, int HDP, bool SIG, bool CAP, int V>
__global__ void __launch_bounds__(AT_DIRECT_WARPS * 32) attn_direct_kernel(const TA* qkv, int row_stride, TA* __restrict__ out, const TA* cache,
                                                                          const int* __restrict__ block_table, int bt_stride, const int* __restrict__ tok_pos,
                                                                          const int* __restrict__ tok_entry, int page_size, int page_shift, int nh, int nkv, int hd,
                                                                          float scale, int window, const float* __restrict__ sink,
                                                                          const float* __restrict__ dist_bias, int dist_far, float cap, int vec) {
    constexpr int NV = (HDP + 63) / 64;
    __shared__ __align__(16) float qs_all[AT_DIRECT_WARPS][HDP], ps_all[AT_DIRECT_WARPS][AT_KEYS];
    il_pdl_wait();
    il_pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x, j = blockIdx.y * AT_DIRECT_WARPS + warp;
    if (j >= nh) return;
    const int g = j / (nh / nkv);
    float* qs = qs_all[warp];
    float* ps = ps_all[warp];
    const TA* qrow = qkv + (size_t)t * row_stride + (size_t)j * hd;
    for (int d = lane; d < HDP; d += 32) qs[d] = d < hd ? il_to_f(qrow[d]) : 0.f;
    const int pos = tok_pos[t];
    const int* bt = block_table + (size_t)tok_entry[t] * bt_stride;
    const int lo = il_mask_lo(pos, window), n_keys = pos - lo + 1, tiles = (n_keys + AT_KEYS - 1) / AT_KEYS;
    const size_t page_elems = (size_t)2 * nkv * page_size * hd, v_off = (size_t)nkv * page_size * hd;
    float m[V], l[V];
    il_f2 acc[V][NV];
#pragma unroll
    for (int u = 0; u < V; ++u) {
        m[u] = -INFINITY, l[u] = 0.f;
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[u][v] = 0ull;
    }
    __syncwarp();
    for (int t0 = 0; t0 < tiles; t0 += V) {
#pragma unroll
        for (int u = 0; u < V; ++u) {             // tile i of the keys goes to running sum i % V
            const int tile = t0 + u;
            if (V > 1 && tile >= tiles) break;
            const int kk = tile * AT_KEYS + lane;
            const bool in = kk < n_keys;
            const int kp = lo + (in ? kk : 0), pi = page_shift >= 0 ? kp >> page_shift : kp / page_size;
            const TA* krow = cache + (size_t)bt[pi] * page_elems + ((size_t)g * page_size + (kp - pi * page_size)) * hd;
            il_f2 s2[2] = {0ull, 0ull};
            if (vec == 2) {
#pragma unroll 4
                for (int d = 0; d < HDP; d += 8) {
                    if (d >= hd) break;
                    il_f2 a[4];
                    at_load8(krow + d, a);
                    const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(qs + d), b1 = *reinterpret_cast<const ulonglong2*>(qs + d + 4);
                    s2[0] = il_f2_fma(a[0], b0.x, s2[0]);
                    s2[1] = il_f2_fma(a[1], b0.y, s2[1]);
                    s2[0] = il_f2_fma(a[2], b1.x, s2[0]);
                    s2[1] = il_f2_fma(a[3], b1.y, s2[1]);
                }
            } else {
#pragma unroll 4
                for (int d = 0; d < HDP; d += 4) {
                    if (d >= hd) break;
                    il_f2 a0, a1;
                    at_load4(krow + d, hd - d, vec, a0, a1);
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(qs + d);
                    s2[0] = il_f2_fma(a0, b.x, s2[0]);
                    s2[1] = il_f2_fma(a1, b.y, s2[1]);
                }
            }
            float d0, d1;
            il_f2_get(il_f2_add(s2[0], s2[1]), d0, d1);
            const float* bias = dist_bias && in ? dist_bias + (size_t)min(n_keys - 1 - kk, dist_far) * nh + j : nullptr;
            ps[lane] = at_weight<SIG, CAP, NV>(d0, d1, in, scale, cap, bias, m[u], l[u], acc[u]);
            __syncwarp();
            const unsigned long long row = reinterpret_cast<unsigned long long>(krow);
            const int n = min(AT_KEYS, n_keys - tile * AT_KEYS);
#pragma unroll 4
            for (int key = 0; key < n; ++key) {
                const TA* vrow = reinterpret_cast<const TA*>(__shfl_sync(0xffffffffu, row, key)) + v_off;
                const il_f2 w = il_f2_dup(ps[key]);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const int d = 2 * lane + 64 * v;
                    if (d < hd) acc[u][v] = il_f2_fma(w, at_load2(vrow + d, hd - d, vec), acc[u][v]);
                }
            }
            __syncwarp();                         // ps is written again in the next tile
        }
    }
    if (!SIG)
#pragma unroll
        for (int u = 0; u < V; ++u) l[u] = il_warp_sum(l[u]);
    if (V > 1) {
        const float m0 = m[0];
#pragma unroll
        for (int u = 1; u < V; ++u) m[0] = fmaxf(m[0], m[u]);
        at_first<SIG, NV>(m0, m[0], l[0], acc[0]);
#pragma unroll
        for (int u = 1; u < V; ++u) {
            const float c = at_factor<SIG>(m[u], m[0]);
            l[0] = __fmaf_rn(c, l[u], l[0]);
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[0][v] = il_f2_fma(il_f2_dup(c), acc[u][v], acc[0][v]);
        }
    }
    at_store<TA, SIG, NV>(out + (size_t)t * nh * hd + (size_t)j * hd, hd, lane, sink ? sink + j : nullptr, m[0], l[0], acc[0]);
}

// Warps that share a head in a block of 8 warps, as many as shared memory holds tiles for; and the running sums of a head: twice as many where
// a block of 16 has the memory. 16 warps for one token, 8 for many: 16 heads on 2 of 64, 2,000 keys 76 and 93 us, 2,048 tokens 889 and 832; 32 on 2 of
// 128, 129 and 153, 2,048 tokens 3,747 and 2,973.
__host__ __device__ constexpr int at_fit(int hdp) { return hdp <= 32 ? 8 : hdp == 64 ? 4 : hdp == 128 ? 2 : 1; }
__host__ __device__ constexpr int at_warps_a_head(int hdp, int HW) { return 8 / HW < at_fit(hdp) ? 8 / HW : at_fit(hdp); }
__host__ __device__ constexpr int at_sums(int hdp, int HW) { return 2 * at_warps_a_head(hdp, HW) <= at_fit(hdp) && 16 / HW >= 2 * at_warps_a_head(hdp, HW) ? 2 * at_warps_a_head(hdp, HW) : at_warps_a_head(hdp, HW); }

static_assert(at_sums(256, 1) == 1 && at_sums(256, 4) == 1 && at_sums(128, 1) == 2 && at_sums(128, 2) == 2 && at_sums(64, 1) == 4 && at_sums(64, 2) == 4 &&
              at_sums(32, 1) == 8, "attn_direct_kernel's sums");

struct AtArgs {
    const void *qkv, *cache;
    void* out;
    const int *block_table, *tok_pos, *tok_entry;
    const float *sink, *dist_bias;
    int row_stride, bt_stride, page_size, T, nh, nkv, hd, window, dist_far;
    float scale, cap;
    cudaStream_t stream;
};

template <typename TA, int HDP, bool SIG, bool CAP, int R>
static cudaError_t at_launch_as(const AtArgs& a, int HW, int n_hb, int KS) {
    int shift = -1;
    if ((a.page_size & (a.page_size - 1)) == 0)
        for (shift = 0; (1 << shift) < a.page_size; ++shift) {}
    const int async = sizeof(TA) == 4 && a.hd % 4 == 0 && !((uintptr_t)a.cache & 15);
    constexpr int smem_max = (2 * at_round_floats(HDP, at_fit(HDP)) + 8 * HDP + 64 * AT_KEYS) * 4;
    const int smem = (2 * at_round_floats(HDP, KS) + HW * HDP + HW * KS * AT_KEYS) * 4;
    static bool done[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !done[dev]) {
        e = cudaFuncSetAttribute(attn_tile_kernel<TA, HDP, SIG, CAP, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    return il_launch(attn_tile_kernel<TA, HDP, SIG, CAP, R>, dim3(a.T, a.nkv * n_hb), dim3(HW * KS * 32), (size_t)smem, a.stream, (const TA*)a.qkv, a.row_stride,
                     (TA*)a.out, (const TA*)a.cache, a.block_table, a.bt_stride, a.tok_pos, a.tok_entry, a.page_size, shift, a.nh, a.nkv, a.hd, a.scale,
                     a.window, a.sink, a.dist_bias, a.dist_far, a.cap, HW, KS, async);
}
template <typename TA, int HDP, bool SIG, bool CAP, int V>
static cudaError_t at_launch_direct(const AtArgs& a) {
    int shift = -1;
    if ((a.page_size & (a.page_size - 1)) == 0)
        for (shift = 0; (1 << shift) < a.page_size; ++shift) {}
    const uintptr_t at = (uintptr_t)a.cache;       // columns of a row that a load may take: 8, 4, 1
    const int vec = a.hd % 8 == 0 && !(at & (8 * sizeof(TA) - 1)) ? 2 : a.hd % 4 == 0 && !(at & (4 * sizeof(TA) - 1)) ? 1 : 0;
    return il_launch(attn_direct_kernel<TA, HDP, SIG, CAP, V>, dim3(a.T, (a.nh + AT_DIRECT_WARPS - 1) / AT_DIRECT_WARPS), dim3(AT_DIRECT_WARPS * 32), (size_t)0,
                     a.stream, (const TA*)a.qkv, a.row_stride, (TA*)a.out, (const TA*)a.cache, a.block_table, a.bt_stride, a.tok_pos, a.tok_entry, a.page_size,
                     shift, a.nh, a.nkv, a.hd, a.scale, a.window, a.sink, a.dist_bias, a.dist_far, a.cap, vec);
}
// Whether a step runs the kernel that stages nothing: where few heads share a kv head and the tiles' blocks, about one an SM there, are so many waves (0: never).
// A long context is a longer chain for its one warp a head than for the tiles' several, so the waves wanted grow with the contexts the block table has room for
// (`keys`), up to 512. bfloat16 tiles are widened by plain loads as they are staged, which float32 leaves to asynchronous copies: fewer waves. Measured, tiles / direct / key by
// key as it was before both, us:
//   float32  256: 8 heads on 8, 1,024 tokens 9,580 / 1,102 / 1,213, 64 single tokens over 500 keys 679 / 658 / 1,013; 8 on 4 3,006 / 1,110 / 1,201; 9 on 3 1,852 / 1,252 / 1,378, 300
//            tokens 200 / 212 / 264; 8 on 2 1,104 / 1,123 / 1,233
//            128: 8 on 8, 1,024 tokens 2,277 / 831 / 1,079, 64 single tokens 164 / 551 / 926; 12 on 12, 64 tokens 41 / 34 / 52; 8 on 4, 1,024 tokens 784 / 837 / 1,079
//            64: 16 on 16, 1,024 tokens 1,421 / 748 / 1,587, 64 single tokens 96 / 305 / 722, 30 tokens 19 / 13 / 24; 16 on 8, 1,024 tokens 647 / 746 / 1,555
//            32: 32 on 32, 1,024 tokens 1,725 / 1,386 / 2,700, after 2,000 cached 5,882 / 6,662 / 12,229, 64 tokens 59 / 21 / 43
//   bfloat16 256: 8 on 8 18,118 / 1,015 / 1,278; 8 on 2 1,733 / 1,066 / 1,267, 300 tokens 189 / 182 / 278    128: 8 on 4 1,462 / 739 / 1,193; 9 on 3, 300 tokens 103 / 154 / 268
//            64: 16 on 8 991 / 683 / 1,759, 64 single tokens 77 / 147 / 377; 9 on 3 322 / 442 / 1,111    32: 32 on 32 2,345 / 1,213 / 2,909; 16 on 8 401 / 621 / 1,570
__host__ __device__ constexpr int at_direct_waves(int hdp, int HW, int bytes) {
    if (bytes == 4) return hdp == 256 ? (HW <= 2 ? 2 : HW == 3 ? 12 : 0) : HW > 1 ? 0 : hdp == 128 ? 10 : hdp == 64 ? 20 : 40;
    return hdp == 256 ? (HW <= 2 ? 2 : HW <= 4 ? HW : 0) : HW > 2 ? 0 : hdp == 128 ? 2 * HW : hdp == 64 ? (HW == 1 ? 4 : 16) : HW == 1 ? 8 : 0;
}
static bool at_direct(int hdp, int HW, int bytes, long long blocks, long long keys) {
    const long long waves = at_direct_waves(hdp, HW, bytes);
    if (waves == 0 || blocks < 148 || (bytes == 4 && hdp == 32 && keys > 1024)) return false;
    return blocks * 512 >= 148 * waves * (keys < 512 ? keys : 512);
}
template <typename TA, int HDP, bool SIG, bool CAP>
static cudaError_t at_launch(const AtArgs& a) {
    const int G = a.nh / a.nkv, HW = G < 8 ? G : 8, n_hb = (G + HW - 1) / HW;
    const long long blocks = (long long)a.T * a.nkv * n_hb;
    const int KS = at_warps_a_head(HDP, HW), sums = at_sums(HDP, HW);
    // (wherever the other kernel is taken a head has at_fit(HDP) running sums)
    if (at_direct(HDP, HW, sizeof(TA), blocks, (long long)a.bt_stride * a.page_size)) return at_launch_direct<TA, HDP, SIG, CAP, at_fit(HDP)>(a);
    // Few (token, kv head) pairs, less than two blocks an SM: a warp for every sum.
    if (sums == KS || blocks < 2 * 148) {
        // Eight heads a block read their tiles from one SM's shared memory, which bounds a round of tiles; where SMs are idle four do (the same
        // sums, so the same bits). 16 heads on 2 of 64, one to eight tokens over 66 / 450 / 2,000 keys, us: 6.3 / 20.2 / 75.6 with eight, 5.3 / 15.7 / 57.4
        // with four, 5.5 / 16.0 / 57.7 with two, whose few threads bring the tiles in more slowly; 32 on 2 of 128: 9.5 / 33.3 / 128.5, 7.9 / 25.9 / 97.5.
        const int hw = HW == 8 && (long long)a.T * a.nkv * ((G + 3) / 4) <= 148 ? 4 : HW;
        return at_launch_as<TA, HDP, SIG, CAP, 1>(a, hw, (G + hw - 1) / hw, sums);
    }
    if constexpr (HDP < 256) return at_launch_as<TA, HDP, SIG, CAP, 2>(a, HW, n_hb, KS);
    return cudaErrorInvalidValue;                 // (not reached: one sum a head at 256)
}
template <typename TA, bool SIG, bool CAP> static cudaError_t at_sizes(const AtArgs& a) {
    return a.hd <= 32 ? at_launch<TA, 32, SIG, CAP>(a) : a.hd <= 64 ? at_launch<TA, 64, SIG, CAP>(a)
         : a.hd <= 128 ? at_launch<TA, 128, SIG, CAP>(a) : at_launch<TA, 256, SIG, CAP>(a);
}
template <typename TA> static cudaError_t at_modes(const AtArgs& a, int sigmoid) {
    return sigmoid ? at_sizes<TA, true, false>(a) : a.cap > 0.f ? at_sizes<TA, false, true>(a) : at_sizes<TA, false, false>(a);
}

// ---- head sizes beyond 256: one warp per (token, query head), keys one by one with an online softmax -------------------------------
// A lane holds head_dim / 32 elements of the query and of the output.
constexpr int AP_MAX_PER_LANE = 32;
template <typename TA, bool SIG, bool CAP>
__global__ void attn_plain_kernel(const TA* __restrict__ qkv, int row_stride, TA* __restrict__ out,
                                  const TA* __restrict__ cache, const int* __restrict__ block_table, int bt_stride,
                                  const int* __restrict__ tok_pos, const int* __restrict__ tok_entry, int page_size,
                                  int nh, int nkv, int hd, float scale, int window, const float* __restrict__ sink,
                                  const float* __restrict__ dist_bias, int dist_far, float cap) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.y * (blockDim.x >> 5) + warp;
    const int t = blockIdx.x;
    if (j >= nh) return;
    const int g = j / (nh / nkv);
    const int pos = tok_pos[t];
    const int* bt = block_table + (size_t)tok_entry[t] * bt_stride;
    const int lo = il_mask_lo(pos, window);

    float q[AP_MAX_PER_LANE], acc[AP_MAX_PER_LANE];
    const TA* qrow = qkv + (size_t)t * row_stride + (size_t)j * hd;
#pragma unroll
    for (int r = 0; r < AP_MAX_PER_LANE; ++r) {
        const int d = lane + 32 * r;
        q[r] = d < hd ? il_to_f(qrow[d]) : 0.f;
        acc[r] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    const size_t page_elems = (size_t)2 * nkv * page_size * hd;
    for (int kp = lo; kp <= pos; ++kp) {
        const int page = bt[kp / page_size];
        const TA* krow = cache + (size_t)page * page_elems + ((size_t)g * page_size + kp % page_size) * hd;
        const TA* vrow = krow + (size_t)nkv * page_size * hd;
        float dot = 0.f;
#pragma unroll
        for (int r = 0; r < AP_MAX_PER_LANE; ++r) {
            const int d = lane + 32 * r;
            if (d < hd) dot += q[r] * il_to_f(krow[d]);
        }
        dot = il_warp_sum(dot) * scale;
        if (CAP) dot = cap * tanhf(dot / cap);
        if (dist_bias) dot += dist_bias[(size_t)min(pos - kp, dist_far) * nh + j];
        if constexpr (SIG) {
            const float w = 1.f / (1.f + expf(-dot));
#pragma unroll
            for (int r = 0; r < AP_MAX_PER_LANE; ++r) {
                const int d = lane + 32 * r;
                if (d < hd) acc[r] = fmaf(w, il_to_f(vrow[d]), acc[r]);
            }
            continue;
        }
        const float mn = fmaxf(m, dot);
        const float corr = expf(m - mn);  // exp(-inf) = 0 on the first key
        const float p = expf(dot - mn);
        l = l * corr + p;
#pragma unroll
        for (int r = 0; r < AP_MAX_PER_LANE; ++r) {
            const int d = lane + 32 * r;
            if (d < hd) acc[r] = acc[r] * corr + p * il_to_f(vrow[d]);
        }
        m = mn;
    }
    TA* orow = out + (size_t)t * nh * hd + (size_t)j * hd;
    if (sink) l += expf(sink[j] - m);             // (+inf when the sink towers over every score: the row is then zero)
    const float inv = SIG ? 1.f : 1.f / l;
#pragma unroll
    for (int r = 0; r < AP_MAX_PER_LANE; ++r) {
        const int d = lane + 32 * r;
        if (d < hd) orow[d] = il_from_f<TA>(acc[r] * inv);
    }
}

IL_EXPORT int il_attn_plain(const void* qkv, int act_kind, int row_stride, void* out, const void* cache,
                            const int* block_table, int bt_stride, const int* tok_pos, const int* tok_entry,
                            int page_size, int T, int nh, int nkv, int hd, float scale, int window,
                            const float* sink, const float* dist_bias, int dist_far, int sigmoid, float cap, cudaStream_t stream) {
    if (T <= 0) return IL_OK;
    if ((dist_bias && dist_far < 0) || (sigmoid && sink) || (cap > 0.f && (sigmoid || dist_bias))) return IL_BAD_ARG;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || page_size <= 0) return IL_BAD_ARG;
    if (hd > 1024) return IL_UNSUPPORTED;
    if (act_kind != IL_F32 && act_kind != IL_BF16) return IL_BAD_ARG;
    if (hd <= 256) {
        const AtArgs a{qkv, cache, out, block_table, tok_pos, tok_entry, sink, dist_bias, row_stride, bt_stride, page_size, T, nh, nkv, hd, window,
                       dist_far, scale, cap, stream};
        const cudaError_t e = act_kind == IL_F32 ? at_modes<float>(a, sigmoid) : at_modes<__nv_bfloat16>(a, sigmoid);
        if (e != cudaSuccess) return 1000 + (int)e;
        IL_LAUNCH_CHECK();
        return IL_OK;
    }
    const int warps = 4;
    dim3 grid(T, (nh + warps - 1) / warps);
#define AP_LAUNCH1(TA, S, C)                                                                                                                     \
    attn_plain_kernel<TA, S, C><<<grid, warps * 32, 0, stream>>>((const TA*)qkv, row_stride, (TA*)out, (const TA*)cache, block_table, bt_stride, \
                                                                 tok_pos, tok_entry, page_size, nh, nkv, hd, scale, window, sink, dist_bias, dist_far, cap)
#define AP_LAUNCH(TA)                                    \
    do {                                                 \
        if (sigmoid) AP_LAUNCH1(TA, true, false);        \
        else if (cap > 0.f) AP_LAUNCH1(TA, false, true); \
        else AP_LAUNCH1(TA, false, false);               \
    } while (0)
    if (act_kind == IL_F32) AP_LAUNCH(float); else AP_LAUNCH(__nv_bfloat16);
#undef AP_LAUNCH
#undef AP_LAUNCH1
    IL_LAUNCH_CHECK();
    return IL_OK;
}
