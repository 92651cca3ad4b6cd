// Rotary position encoding of q and k in place (rotate-half pairing (i, i + rot/2)), then the
// write of the rotated k and of v into the paged cache. Angles are pos * inv_freq[i] in f32;
// cos and sin are multiplied by `mscale` (1 unless a LongRoPE configuration extends the context).
//
// qkv row layout: [nh heads of q | nkv heads of k | nkv heads of v], each head_dim wide.
// Cache layout of one layer: [page][0=K,1=V][kv head][slot in page][head_dim].
// A token's slot follows from its entry's block-table row and its absolute position.
#include "common.cuh"

__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 ld2(const __nv_bfloat16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }
__device__ __forceinline__ void st2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ void st2(__nv_bfloat16* p, float2 v) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(v.x, v.y); }

template <typename TA>
__global__ void rope_store_kernel(TA* __restrict__ qkv, int row_stride, const int* __restrict__ tok_pos,
                                  const int* __restrict__ tok_entry, const int* __restrict__ block_table,
                                  int bt_stride, TA* __restrict__ cache, int page_size, int nh, int nkv, int hd,
                                  int rot, const float* __restrict__ inv_freq, float mscale) {
    // Positions, block tables and the angle table do not come from the kernel before this one: all of that is done
    // before waiting for it. After the wait a thread reads its pairs once and writes them where they go: q and k back
    // into the row, k and v into the cache slot.
    const int t = blockIdx.x;
    const int pos = tok_pos[t];
    TA* row = qkv + (size_t)t * row_stride;
    const int half = rot >> 1;
    __shared__ float cs[128], sn[128];            // rot <= head_dim <= 256
    TA* kdst = nullptr;                           // this token's K slot of kv head 0, or null: nothing to store
    size_t head_step = 0, v_off = 0;
    if (cache) {
        const int e = tok_entry[t];
        const int page = block_table[(size_t)e * bt_stride + pos / page_size];
        if (page >= 0) {                          // the host reserves every page a step touches; never write elsewhere
            head_step = (size_t)page_size * hd;
            v_off = (size_t)nkv * head_step;
            kdst = cache + (size_t)page * 2 * v_off + (size_t)(pos % page_size) * hd;
        }
    }
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float s, c;
        sincosf((float)pos * inv_freq[i], &s, &c);
        sn[i] = s * mscale;
        cs[i] = c * mscale;
    }
    __syncthreads();
    il_pdl_launch_dependents();                   // the attention kernel behind this one has a prologue of its own to run meanwhile
    il_pdl_wait();
    // After the wait every load of a batch is issued before its first store: the row is read and written in place, so
    // the compiler keeps loads behind earlier stores, and a loop of load-rotate-store rounds would pay the memory
    // latency once per round.
    constexpr int VEC = 16 / sizeof(TA);          // elements per 16-byte chunk; head_dim is a multiple of 16
    const int cpr = hd / VEC;
    const TA* ksrc = row + (size_t)nh * hd;
    const TA* vsrc = ksrc + (size_t)nkv * hd;
    constexpr int UV = 2, UR = 4;
    for (int vb = 0; vb < (kdst ? nkv * cpr : 0) || vb == 0; vb += UV * blockDim.x) {
        uint4 vv[UV];
        const int n_v = kdst ? nkv * cpr : 0;
#pragma unroll
        for (int u = 0; u < UV; ++u) {
            const int idx = vb + u * blockDim.x + threadIdx.x;
            if (idx < n_v) vv[u] = *reinterpret_cast<const uint4*>(vsrc + (size_t)(idx / cpr) * hd + (size_t)(idx % cpr) * VEC);
        }
        if (vb == 0 && half > 0) {
            if ((half & 1) == 0) {                // two neighbouring pairs per thread, 4- or 8-byte accesses
                const int hp = half >> 1, n2 = (nh + nkv) * hp;
                for (int rb = 0; rb < n2; rb += UR * blockDim.x) {
                    float2 a[UR], b[UR];
#pragma unroll
                    for (int u = 0; u < UR; ++u) {
                        const int idx = rb + u * blockDim.x + threadIdx.x;
                        if (idx < n2) {
                            const int j = idx / hp, i = (idx - j * hp) * 2;
                            a[u] = ld2(row + (size_t)j * hd + i);
                            b[u] = ld2(row + (size_t)j * hd + i + half);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < UR; ++u) {
                        const int idx = rb + u * blockDim.x + threadIdx.x;
                        if (idx < n2) {
                            const int j = idx / hp, i = (idx - j * hp) * 2;
                            TA* base = row + (size_t)j * hd;
                            const float s0 = sn[i], c0 = cs[i], s1 = sn[i + 1], c1 = cs[i + 1];
                            const float2 lo = make_float2(a[u].x * c0 - b[u].x * s0, a[u].y * c1 - b[u].y * s1);
                            const float2 hi = make_float2(b[u].x * c0 + a[u].x * s0, b[u].y * c1 + a[u].y * s1);
                            st2(base + i, lo);
                            st2(base + i + half, hi);
                            if (j >= nh && kdst) {
                                TA* kd = kdst + (size_t)(j - nh) * head_step;
                                st2(kd + i, lo);
                                st2(kd + i + half, hi);
                            }
                        }
                    }
                }
            } else {
                const int n_pairs = (nh + nkv) * half;
                for (int idx = threadIdx.x; idx < n_pairs; idx += blockDim.x) {
                    const int j = idx / half, i = idx - j * half;
                    TA* base = row + (size_t)j * hd;
                    const float s = sn[i], c = cs[i];
                    const float x1 = il_to_f(base[i]), x2 = il_to_f(base[i + half]);
                    const TA lo = il_from_f<TA>(x1 * c - x2 * s), hi = il_from_f<TA>(x2 * c + x1 * s);
                    base[i] = lo;
                    base[i + half] = hi;
                    if (j >= nh && kdst) {
                        TA* kd = kdst + (size_t)(j - nh) * head_step;
                        kd[i] = lo;
                        kd[i + half] = hi;
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < UV; ++u) {
            const int idx = vb + u * blockDim.x + threadIdx.x;
            if (idx < n_v)
                *reinterpret_cast<uint4*>(kdst + v_off + (size_t)(idx / cpr) * head_step + (size_t)(idx % cpr) * VEC) = vv[u];
        }
    }
    if (!kdst) return;
    // what the rotation did not touch of k: the dimensions beyond rot (none when rot == head_dim)
    const int tail = hd - rot;
    for (int idx = threadIdx.x; idx < nkv * tail; idx += blockDim.x) {
        const int g = idx / tail, c = rot + (idx - g * tail);
        kdst[(size_t)g * head_step + c] = ksrc[(size_t)g * hd + c];
    }
}

// A pair of a prompt portion rotated, x1 c - x2 s and x2 c + x1 s, written out in the rounding that both kernels for many tokens have: the products
// x2 s and x2 c are rounded first. (Left to the compiler, the one below and the one in 16-byte pieces differed in bfloat16. The kernel for few tokens
// rounds x1 s instead of x2 c.)
__device__ __forceinline__ float rope_lo(float x1, float x2, float c, float s) { return __fmaf_rn(x1, c, -__fmul_rn(x2, s)); }
__device__ __forceinline__ float rope_hi(float x1, float x2, float c, float s) { return __fmaf_rn(x1, s, __fmul_rn(x2, c)); }

// The same for many tokens (prompt portions) where the pairs are not whole 16-byte pieces: a block's latency does not matter there, how many blocks an SM holds
// does; two passes (rotate in place, then copy k and v to the cache in 16-byte pieces), 256 threads, few registers.
template <typename TA>
__global__ void rope_store_many_kernel(TA* __restrict__ qkv, int row_stride, const int* __restrict__ tok_pos,
                                  const int* __restrict__ tok_entry, const int* __restrict__ block_table,
                                  int bt_stride, TA* __restrict__ cache, int page_size, int nh, int nkv, int hd,
                                  int rot, const float* __restrict__ inv_freq, float mscale) {
    il_pdl_begin();
    const int t = blockIdx.x;
    const int pos = tok_pos[t];
    TA* row = qkv + (size_t)t * row_stride;
    const int half = rot >> 1;
    __shared__ float cs[128], sn[128];            // rot <= head_dim <= 256
    if (half > 0) {
        for (int i = threadIdx.x; i < half; i += blockDim.x) {
            float s, c;
            sincosf((float)pos * inv_freq[i], &s, &c);
            sn[i] = s * mscale;
            cs[i] = c * mscale;
        }
        __syncthreads();
        if ((half & 1) == 0) {                    // two neighbouring pairs per thread, 4- or 8-byte accesses
            const int hp = half >> 1, n2 = (nh + nkv) * hp;
            for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
                const int j = idx / hp, i = (idx - j * hp) * 2;
                TA* base = row + (size_t)j * hd;
                const float2 a = ld2(base + i), b = ld2(base + i + half);
                const float s0 = sn[i], c0 = cs[i], s1 = sn[i + 1], c1 = cs[i + 1];
                st2(base + i, make_float2(rope_lo(a.x, b.x, c0, s0), rope_lo(a.y, b.y, c1, s1)));
                st2(base + i + half, make_float2(rope_hi(a.x, b.x, c0, s0), rope_hi(a.y, b.y, c1, s1)));
            }
        } else {
            const int n_pairs = (nh + nkv) * half;
            for (int idx = threadIdx.x; idx < n_pairs; idx += blockDim.x) {
                const int j = idx / half, i = idx - j * half;
                TA* base = row + (size_t)j * hd;
                const float s = sn[i], c = cs[i];
                const float x1 = il_to_f(base[i]), x2 = il_to_f(base[i + half]);
                base[i] = il_from_f<TA>(x1 * c - x2 * s);
                base[i + half] = il_from_f<TA>(x2 * c + x1 * s);
            }
        }
    }
    if (!cache) return;
    __syncthreads();
    const int e = tok_entry[t];
    const int page = block_table[(size_t)e * bt_stride + pos / page_size];
    if (page < 0) return;  // the host reserves every page a step touches; never write elsewhere
    const int off = pos % page_size;
    const TA* ksrc = row + (size_t)nh * hd;
    const TA* vsrc = ksrc + (size_t)nkv * hd;
    const size_t page_elems = (size_t)2 * nkv * page_size * hd;
    TA* kdst = cache + (size_t)page * page_elems;
    TA* vdst = kdst + (size_t)nkv * page_size * hd;
    constexpr int VEC = 16 / sizeof(TA);          // elements per 16-byte chunk; head_dim is a multiple of 16
    const int cpr = hd / VEC;
    for (int idx = threadIdx.x; idx < nkv * cpr; idx += blockDim.x) {
        const int g = idx / cpr, c = idx - g * cpr;
        const size_t o = ((size_t)g * page_size + off) * hd + (size_t)c * VEC;
        *reinterpret_cast<uint4*>(kdst + o) = *reinterpret_cast<const uint4*>(ksrc + (size_t)g * hd + (size_t)c * VEC);
        *reinterpret_cast<uint4*>(vdst + o) = *reinterpret_cast<const uint4*>(vsrc + (size_t)g * hd + (size_t)c * VEC);
    }
}

// The same where the rotated pairs come in whole 16-byte pieces: one pass, a thread an item (a piece of the first half of a
// rotated head and the piece it pairs with, a piece of v, or a piece of k that is not rotated), several tokens a block where a
// token has few items. The row has just been written and lies in the L2, so what bounds it is loads in flight: the first of a
// thread are asked for before the angles are computed (8B sizes, 2,048 tokens, without that 10.5 us).
// Two passes before / so, us: 32 heads on 2 of 128 bfloat16, 600 / 2,048 / 8,192 tokens 4.2 / 9.2 / 32.1 and 3.6 / 8.1 / 27.4; 16 on 2 of 64 2.9 / 5.7 /
// 16.5 and 2.7 / 3.5 / 9.9; the same in float32 2.9 / 5.7 / 16.4 and 2.9 / 5.3 / 15.8; 65 tokens 2.4 to 3.1 and 2.3 to 2.4.
constexpr int ROPE_WIDE_TOKENS = 8;
template <typename TA>
__global__ void __launch_bounds__(512) rope_store_wide_kernel(TA* qkv, int row_stride, const int* tok_pos, const int* tok_entry, const int* block_table, int bt_stride,
                                                              TA* cache, int page_size, int T, int nh, int nkv, int hd, int rot, const float* inv_freq, float mscale,
                                                              int tokens, int items) {
    constexpr int VEC = 16 / sizeof(TA);
    __shared__ __align__(16) float cs[ROPE_WIDE_TOKENS * 128], sn[ROPE_WIDE_TOKENS * 128];        // rot <= head_dim <= 256
    __shared__ TA* slot[ROPE_WIDE_TOKENS];        // a token's K slot of kv head 0, or null: nothing to store
    const int t0 = blockIdx.x * tokens, n = min(tokens, T - t0), half = rot >> 1;
    const size_t head_step = (size_t)page_size * hd;
    const int hp = half / VEC, n_rot = (nh + nkv) * hp, cpr = hd / VEC, tail = (hd - rot) / VEC;
    struct Item { TA* from; int tok, head, i, step; };      // step: columns to the piece it is rotated with, 0: none, it is copied; i: its column in a slot
    const auto item = [&](int idx) {
        Item it;
        it.tok = idx / items;
        int k = idx - it.tok * items;
        TA* const row = qkv + (size_t)(t0 + it.tok) * row_stride;
        if (k < n_rot) {
            const int j = k / hp;
            it.i = (k - j * hp) * VEC, it.head = j - nh, it.step = half;
            it.from = row + (size_t)j * hd + it.i;
        } else {                                  // v (kv heads nkv .. 2 nkv - 1), then what the rotation does not touch of k
            k -= n_rot;
            const bool v = k < nkv * cpr;
            if (!v) k -= nkv * cpr;
            const int per = v ? cpr : tail, g = k / per;
            it.i = (v ? 0 : rot) + (k - g * per) * VEC, it.head = (v ? nkv : 0) + g, it.step = 0;
            it.from = row + (size_t)(nh + it.head) * hd + it.i;
        }
        return it;
    };
    il_pdl_begin();
    // the first item's pieces are on their way while the angles are computed
    int idx = threadIdx.x;
    Item it;
    uint4 a, b;
    if (idx < n * items) {
        it = item(idx);
        a = *reinterpret_cast<const uint4*>(it.from);
        if (it.step) b = *reinterpret_cast<const uint4*>(it.from + half);
    }
    for (int i = threadIdx.x; i < n * half; i += blockDim.x) {
        const int tok = i / half;
        float s, c;
        sincosf((float)tok_pos[t0 + tok] * inv_freq[i - tok * half], &s, &c);
        sn[i] = s * mscale;
        cs[i] = c * mscale;
    }
    if (threadIdx.x < n) {
        TA* at = nullptr;
        if (cache) {
            const int pos = tok_pos[t0 + threadIdx.x], page = block_table[(size_t)tok_entry[t0 + threadIdx.x] * bt_stride + pos / page_size];
            if (page >= 0) at = cache + (size_t)page * 2 * nkv * head_step + (size_t)(pos % page_size) * hd;     // the host reserves every page a step touches
        }
        slot[threadIdx.x] = at;
    }
    __syncthreads();
    while (idx < n * items) {
        TA* const at = slot[it.tok];
        TA* const to = at + (size_t)it.head * head_step + it.i;       // (K's heads, then V's)
        if (it.step) {
            TA *ap = reinterpret_cast<TA*>(&a), *bp = reinterpret_cast<TA*>(&b);
            const float *c = cs + it.tok * half + it.i, *s = sn + it.tok * half + it.i;
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                const float x1 = il_to_f(ap[e]), x2 = il_to_f(bp[e]);
                ap[e] = il_from_f<TA>(rope_lo(x1, x2, c[e], s[e]));
                bp[e] = il_from_f<TA>(rope_hi(x1, x2, c[e], s[e]));
            }
            *reinterpret_cast<uint4*>(it.from) = a;
            *reinterpret_cast<uint4*>(it.from + half) = b;
            if (it.head >= 0 && at) {
                *reinterpret_cast<uint4*>(to) = a;
                *reinterpret_cast<uint4*>(to + half) = b;
            }
        } else if (at) {
            *reinterpret_cast<uint4*>(to) = a;
        }
        idx += blockDim.x;
        if (idx < n * items) {
            it = item(idx);
            a = *reinterpret_cast<const uint4*>(it.from);
            if (it.step) b = *reinterpret_cast<const uint4*>(it.from + half);
        }
    }
}
template <typename TA>
static int rope_store_wide(void* qkv, int row_stride, const int* tok_pos, const int* tok_entry, const int* block_table, int bt_stride, void* cache, int page_size, int T,
                           int nh, int nkv, int hd, int rot, const float* inv_freq, float mscale, cudaStream_t stream) {
    constexpr int VEC = 16 / sizeof(TA);
    const int items = (nh + nkv) * (rot / 2 / VEC) + (cache ? nkv * ((2 * hd - rot) / VEC) : 0);
    if (items == 0) return IL_OK;
    const int tokens = items > 256 / 2 ? 1 : min(256 / items, ROPE_WIDE_TOKENS), threads = min((tokens * items + 31) / 32 * 32, 512);
    IL_LAUNCH(rope_store_wide_kernel<TA>, (T + tokens - 1) / tokens, threads, 0, stream, (TA*)qkv, row_stride, tok_pos, tok_entry, block_table, bt_stride, (TA*)cache,
              page_size, T, nh, nkv, hd, rot, inv_freq, mscale, tokens, items);
    IL_LAUNCH_CHECK();
    return IL_OK;
}

IL_EXPORT int il_rope_store(void* qkv, int act_kind, int row_stride, const int* tok_pos, const int* tok_entry,
                            const int* block_table, int bt_stride, void* cache, int page_size, int T, int nh,
                            int nkv, int hd, int rot, const float* inv_freq, float mscale, cudaStream_t stream) {
    if (T <= 0) return IL_OK;
    if (hd > 256) return IL_UNSUPPORTED;
    if (nh <= 0 || nkv <= 0 || hd <= 0 || rot < 0 || rot > hd || (rot & 1) || page_size <= 0) return IL_BAD_ARG;
    if (row_stride < (nh + 2 * nkv) * hd || hd % 16 != 0 || row_stride % 8 != 0) return IL_BAD_ARG;
    constexpr int MANY = 64;                      // from here on: the two-pass kernel for throughput
    if (T > MANY) {
        const int vec = act_kind == IL_F32 ? 4 : 8;
        if ((act_kind == IL_F32 || act_kind == IL_BF16) && rot % (2 * vec) == 0 && !(((uintptr_t)qkv | (uintptr_t)cache) & 15)) {
            const auto wide = act_kind == IL_F32 ? rope_store_wide<float> : rope_store_wide<__nv_bfloat16>;
            return wide(qkv, row_stride, tok_pos, tok_entry, block_table, bt_stride, cache, page_size, T, nh, nkv, hd, rot, inv_freq, mscale, stream);
        }
        if (act_kind == IL_F32)
            IL_LAUNCH(rope_store_many_kernel<float>, T, 256, 0, stream, (float*)qkv, row_stride, tok_pos, tok_entry, block_table, bt_stride,
                      (float*)cache, page_size, nh, nkv, hd, rot, inv_freq, mscale);
        else if (act_kind == IL_BF16)
            IL_LAUNCH(rope_store_many_kernel<__nv_bfloat16>, T, 256, 0, stream, (__nv_bfloat16*)qkv, row_stride, tok_pos, tok_entry,
                      block_table, bt_stride, (__nv_bfloat16*)cache, page_size, nh, nkv, hd, rot, inv_freq, mscale);
        else
            return IL_BAD_ARG;
        IL_LAUNCH_CHECK();
        return IL_OK;
    }
    // a thread takes up to four pairs of neighbours at once: enough threads that one round covers a row
    const int pairs2 = (nh + nkv) * (rot / 4);
    int threads = ((pairs2 + 3) / 4 + 31) / 32 * 32;
    threads = threads < 128 ? 128 : (threads > 1024 ? 1024 : threads);
    if (act_kind == IL_F32)
        IL_LAUNCH(rope_store_kernel<float>, T, threads, 0, stream, (float*)qkv, row_stride, tok_pos, tok_entry, block_table, bt_stride,
                  (float*)cache, page_size, nh, nkv, hd, rot, inv_freq, mscale);
    else if (act_kind == IL_BF16)
        IL_LAUNCH(rope_store_kernel<__nv_bfloat16>, T, threads, 0, stream, (__nv_bfloat16*)qkv, row_stride, tok_pos, tok_entry, block_table,
                  bt_stride, (__nv_bfloat16*)cache, page_size, nh, nkv, hd, rot, inv_freq, mscale);
    else
        return IL_BAD_ARG;
    IL_LAUNCH_CHECK();
    return IL_OK;
}
