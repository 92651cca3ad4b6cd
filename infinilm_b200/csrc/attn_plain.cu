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
            // (roundings spelled out: the same bits from both forms of this kernel)
            float s = __fmul_rn(__fadd_rn(d0, d1), scale);
            if (CAP) s = __fmul_rn(cap, tanhf(__fdiv_rn(s, cap)));
            if (dist_bias && in) s = __fadd_rn(s, dist_bias[(size_t)min(n_keys - 1 - kk, dist_far) * nh + j]);
            float p;
            if constexpr (SIG) {
                p = in ? __fdiv_rn(1.f, __fadd_rn(1.f, expf(-s))) : 0.f;
            } else {
                const float mn = fmaxf(m[u], il_warp_max(in ? s : -INFINITY));
                // exp(-inf) = 0 on the first tile; a tile whose scores are all -inf (a bias that masks) leaves the sum as it is
                const float ref = mn == -INFINITY ? 0.f : mn;
                const float corr = mn == -INFINITY ? 1.f : expf(__fadd_rn(m[u], -mn));
                p = in ? expf(__fadd_rn(s, -ref)) : 0.f;
                l[u] = __fmaf_rn(l[u], corr, p);
                m[u] = mn;
                const il_f2 c2 = il_f2_dup(corr);
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[u][v] = il_f2_mul(acc[u][v], c2);
            }
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
        if (!SIG) {
            const float c = m0 == -INFINITY ? 0.f : expf(__fadd_rn(m0, -m[0]));
            l[0] = __fmul_rn(l[0], c);
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[0][v] = il_f2_mul(acc[0][v], il_f2_dup(c));
        }
        for (int i = 1; i < R * KS; ++i) {
            const float* other = sm + (size_t)(i * HW + hs) * (HDP + 4);
            const float mi = other[HDP];
            const float c = SIG ? 1.f : mi == -INFINITY ? 0.f : expf(__fadd_rn(mi, -m[0]));
            l[0] = __fmaf_rn(c, other[HDP + 1], l[0]);
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (HDP >= 64 || 2 * lane < HDP)
                    acc[0][v] = il_f2_fma(il_f2_dup(c), *reinterpret_cast<const il_f2*>(other + 2 * lane + 64 * v), acc[0][v]);
        }
    }
    if (!live) return;
    if (sink) l[0] = __fadd_rn(l[0], expf(__fadd_rn(sink[j], -m[0])));   // (+inf when the sink towers over every score: the row is then zero)
    const float inv = SIG ? 1.f : __fdiv_rn(1.f, l[0]);
    TA* orow = out + (size_t)t * nh * hd + (size_t)j * hd;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        float a, b;
        il_f2_get(acc[0][v], a, b);
        const int d = 2 * lane + 64 * v;
        if (d < hd) orow[d] = il_from_f<TA>(a * inv);
        if (d + 1 < hd) orow[d + 1] = il_from_f<TA>(b * inv);
    }
}

// Warps that share a head in a block of 8 warps, as many as shared memory holds tiles for; and the running sums of a head: twice as many where
// a block of 16 has the memory. 16 warps for one token, 8 for many: 16 heads on 2 of 64, 2,000 keys 76 and 93 us, 2,048 tokens 889 and 832; 32 on 2 of
// 128, 129 and 153, 2,048 tokens 3,747 and 2,973.
__host__ __device__ constexpr int at_fit(int hdp) { return hdp <= 32 ? 8 : hdp == 64 ? 4 : hdp == 128 ? 2 : 1; }
__host__ __device__ constexpr int at_warps_a_head(int hdp, int HW) { return 8 / HW < at_fit(hdp) ? 8 / HW : at_fit(hdp); }
__host__ __device__ constexpr int at_sums(int hdp, int HW) { return 2 * at_warps_a_head(hdp, HW) <= at_fit(hdp) && 16 / HW >= 2 * at_warps_a_head(hdp, HW) ? 2 * at_warps_a_head(hdp, HW) : at_warps_a_head(hdp, HW); }

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
template <typename TA, int HDP, bool SIG, bool CAP>
static cudaError_t at_launch(const AtArgs& a) {
    const int G = a.nh / a.nkv, HW = G < 8 ? G : 8, n_hb = (G + HW - 1) / HW;
    const long long blocks = (long long)a.T * a.nkv * n_hb;
    const int KS = at_warps_a_head(HDP, HW), sums = at_sums(HDP, HW);
    // Few (token, kv head) pairs, less than two blocks an SM: a warp for every sum.
    if (sums == KS || blocks < 2 * 148) return at_launch_as<TA, HDP, SIG, CAP, 1>(a, HW, n_hb, sums);
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
