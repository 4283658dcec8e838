// Top-k mixture-of-experts feed-forward: router (fp32 logits, top-k, softmax over the chosen), grouping of the
// (token, choice) pairs by expert on the device, the two grouped products and the weighted combination.
//
// The pairs of one expert occupy whole 32-row tiles of a sorted row list, so every CTA of the grouped products reads
// ONE expert's weights; rows are gathered from / scattered to token order through the list.  Each output row is a sum
// over the reduction index in a fixed order and the combination adds a token's choices in choice order, so a token's
// result does not depend on which other tokens are in the batch.  bfloat16 products run on the tensor cores
// (blocks_moe_tc.cu); the kernel here serves fp32 and rows that are no multiple of 16 bytes.
#include "blocks_moe.cuh"

namespace tlb {

constexpr int kTileRows = TLB_MOE_TILE_ROWS;

__device__ __forceinline__ float moe_act(float z, int act) {
    return act == 2 ? (z > 0.f ? z * z : 0.f) : act_apply(z, act);  // 2: squared ReLU
}

// W consecutive entries of a row as floats.
template <int W>
__device__ __forceinline__ void moe_load(const float *p, float (&x)[W]) {
    if constexpr (W == 1) x[0] = p[0];
    else {
        const float4 v = load4(p);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
    }
}
template <int W>
__device__ __forceinline__ void moe_load(const bf16 *p, float (&x)[W]) {
    if constexpr (W == 1) x[0] = to_f(p[0]);
    else {
        const uint4 u = *reinterpret_cast<const uint4 *>(p);
        const uint32_t c[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = tl::unpack2<bf16>(c[i]);
            x[2 * i] = f.x, x[2 * i + 1] = f.y;
        }
    }
}

template <typename T, int W>
struct __align__(W * sizeof(T)) MoePiece {
    T v[W];
};

// A CTA routes TOK tokens, so that a row of weights is fetched once for all of them: their rows of h are staged in shared memory,
// the warps share the experts, ROWS rows of weights in flight each (a logit is one warp's dot product in a lane order fixed by the
// width, whatever TOK and the launch are), then warp i picks token i's top-k.  W: entries per access (16 bytes where rows allow).
// aux_w: one more row of weights that is no router output; aux[t] = sigmoid(aux_w . h_t) (the gate of a shared expert).
// Eight tokens a CTA are bound by the fp32 multiply-adds (268 M for 2048 tokens and 64 rows of 2048: 7.5 us): 32 of them a weight entry unpacked, the
// tokens' entries unpacked once, at staging, the two halves of a lane's eight entries in separate planes so that its reads meet no bank conflict (2048
// tokens 36 -> 27 us, 1024 48 -> 19; it was four tokens a CTA, unpacked by every warp).
template <typename T, int TOK, int ROWS, int W>
__global__ void __launch_bounds__(TOK == 1 ? 512 : 256, TOK == 1 ? 1 : 2)
moe_route_kernel(const T *__restrict__ h, const T *__restrict__ w, const T *__restrict__ b, int tokens, int dim, int experts, int top, int scoring,
                 const T *__restrict__ choice_bias, float weight_scale, int group_count, int group_keep, const T *__restrict__ aux_w,
                 float *__restrict__ aux, int32_t *__restrict__ idx, float *__restrict__ gate) {
    extern __shared__ __align__(16) unsigned char route_smem[];
    using X = std::conditional_t<TOK == 1, T, float>;
    constexpr bool PLANES = sizeof(X) * W > 16;  // float entries, eight an access
    X *x = reinterpret_cast<X *>(route_smem);  // [TOK][dim]
    float *logits = reinterpret_cast<float *>(route_smem + (((size_t)TOK * dim * sizeof(X) + 15) & ~(size_t)15));
    const int per_token = 2 * experts + group_count;  // [TOK][..]: see below
    const int t0 = blockIdx.x * TOK, here = min(TOK, tokens - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int d = threadIdx.x * W; d < here * dim; d += blockDim.x * W) {
        if constexpr (PLANES) {  // entries 8 i .. 8 i + 3 of a row in its first half, 8 i + 4 .. 8 i + 7 in its second
            float v[W];
            moe_load<W>(h + (size_t)t0 * dim + d, v);
            float *to = x + d / dim * dim + d % dim / 2;
            *reinterpret_cast<float4 *>(to) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4 *>(to + dim / 2) = make_float4(v[4], v[5], v[6], v[7]);
        } else if constexpr (W == 1) {
            x[d] = from_f<X>(to_f(h[(size_t)t0 * dim + d]));
        } else {
            *reinterpret_cast<uint4 *>(x + d) = *reinterpret_cast<const uint4 *>(h + (size_t)t0 * dim + d);
        }
    }
    if (TOK > 1)  // of tokens that are not there: read below, not used
        for (int d = here * dim + threadIdx.x; d < TOK * dim; d += blockDim.x) x[d] = from_f<X>(0.f);
    __syncthreads();
    const int outputs = experts + (aux_w ? 1 : 0);
    for (int e0 = warp; e0 < outputs; e0 += warps * ROWS) {
        float acc[ROWS][TOK];
        const T *row[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int e = e0 + r * warps;
            // past the last one: the last, not used (a condition in the loops below would keep the rows' chains from overlapping)
            row[r] = e < experts ? w + (size_t)e * dim : aux_w ? aux_w : w + (size_t)(experts - 1) * dim;
#pragma unroll
            for (int i = 0; i < TOK; ++i) acc[r][i] = 0.f;
        }
        // steps of weights on their way while one is used (16 tokens: one 14 us, two 11; 1024 tokens, eight a CTA: one 18.5, two 20)
        constexpr int AHEAD = TOK == 1 ? 2 : 1;
        MoePiece<T, W> next[AHEAD][ROWS];
        auto fetch = [&](int d, MoePiece<T, W> (&to)[ROWS]) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
                if (d < dim) to[r] = *reinterpret_cast<const MoePiece<T, W> *>(row[r] + d);
        };
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) fetch((u * 32 + lane) * W, next[u]);
        for (int d0 = lane * W; d0 < dim; d0 += AHEAD * 32 * W) {
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int d = d0 + u * 32 * W;
                if (d >= dim) break;
                float wv[ROWS][W];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) moe_load<W>(next[u][r].v, wv[r]);
                fetch(d + AHEAD * 32 * W, next[u]);
#pragma unroll
                for (int i = 0; i < TOK; ++i) {
                    float xv[W];
                    if constexpr (PLANES) {
                        const float *from = x + (size_t)i * dim + d / 2;
                        const float4 lo = load4(from), hi = load4(from + dim / 2);
                        xv[0] = lo.x, xv[1] = lo.y, xv[2] = lo.z, xv[3] = lo.w, xv[4] = hi.x, xv[5] = hi.y, xv[6] = hi.z, xv[7] = hi.w;
                    } else {
                        moe_load<W>(x + (size_t)i * dim + d, xv);
                    }
#pragma unroll
                    for (int j = 0; j < W; ++j)
#pragma unroll
                        for (int r = 0; r < ROWS; ++r) acc[r][i] = fmaf(xv[j], wv[r][j], acc[r][i]);
                }
            }
        }
        // the sums one after another, then a lane each to write them: with a bias fetched and a store made behind every sum a CTA of eight
        // tokens waited out 64 round trips (25 us)
        float mine = 0.f;
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int i = 0; i < TOK; ++i) {
                const float s = warp_sum(acc[r][i]);
                if (lane == r * TOK + i) mine = s;
            }
        const int e = e0 + lane / TOK * warps, i = lane % TOK;
        if (lane < ROWS * TOK && e < outputs && i < here) {
            if (e < experts) logits[i * per_token + e] = mine + (b ? to_f(b[e]) : 0.f);
            else aux[t0 + i] = sigmoid(mine);
        }
    }
    __syncthreads();
    if (warp >= here) return;
    const int t = t0 + warp;
    float *z = logits + warp * per_token;  // [experts]: what the choice is made by
    float *p_all = z + experts;            // [experts]: scoring 2, the softmax over all outputs
    float *best = p_all + experts;         // [group_count]: the largest choice score of every group
    if (scoring == 2) {  // scores = softmax over ALL outputs; the choice adds a bias to them, the weights do not
        float m = -INFINITY, sum = 0.f;
        for (int e = lane; e < experts; e += 32) m = fmaxf(m, z[e]);
        m = warp_max(m);
        for (int e = lane; e < experts; e += 32) sum += expf(z[e] - m);
        sum = warp_sum(sum);
        for (int e = lane; e < experts; e += 32) {
            float p = expf(z[e] - m) / sum;
            p_all[e] = p;
            z[e] = p + (choice_bias ? to_f(choice_bias[e]) : 0.f);
        }
        __syncwarp();
    }
    if (group_keep > 0 && group_keep < group_count) {  // only the outputs of the best groups of neighbours can be chosen
        const int size = experts / group_count;
        for (int j = lane; j < group_count; j += 32) {
            float m = -INFINITY;
            for (int e = j * size; e < (j + 1) * size; ++e) m = fmaxf(m, z[e]);
            best[j] = m;
        }
        __syncwarp();
        for (int e = lane; e < experts; e += 32) {
            const int j = e / size;
            int ahead = 0;  // groups in front of this one (lower index wins a tie)
            for (int i = 0; i < group_count; ++i) ahead += best[i] > best[j] || (best[i] == best[j] && i < j);
            if (ahead >= group_keep) z[e] = -INFINITY;
        }
        __syncwarp();
    }
    // top-k by repeated arg-max over the warp (lower index wins a tie); weights = softmax over the chosen logits
    float first_v = 0.f, denom = 0.f;
    for (int k = 0; k < top; ++k) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < experts; e += 32) {
            float v = z[e];
            if (v > bv || (v == bv && e < bi)) bv = v, bi = e;
        }
        for (int o = 16; o > 0; o >>= 1) {
            float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
        }
        if (k == 0) first_v = bv;
        // scoring 0: softmax over the chosen logits (the first choice is the largest); 1: each choice's own sigmoid, as it is
        float p = scoring == 1 ? 1.0f / (1.0f + expf(-bv)) : scoring == 2 ? p_all[min(bi, experts - 1)] : expf(bv - first_v);
        denom += p;
        if (lane == 0) {
            idx[(size_t)t * top + k] = bi;
            gate[(size_t)t * top + k] = p;
            if (bi != 0x7fffffff) z[bi] = -INFINITY;
        }
        __syncwarp();
    }
    if (scoring == 1) return;
    // scoring 2: the chosen scores renormalised (a guard against an all-zero choice) and scaled
    for (int k = lane; k < top; k += 32)
        gate[(size_t)t * top + k] = scoring == 2 ? gate[(size_t)t * top + k] / (denom + 1e-20f) * weight_scale : gate[(size_t)t * top + k] / denom;
}

// C tile [32 rows x 64 columns] of  A[rows, K] . W[e][cols, K]^T, fp32 accumulation in k order.
// 256 threads: thread (ty, tx) owns rows 2 ty .. 2 ty + 1 and columns tx + 16 c, c = 0..3.
constexpr int kBN = 64, kBK = 16;

template <typename T, bool GATED>
__global__ void __launch_bounds__(256)
moe_grouped_kernel(const T *__restrict__ a, const T *__restrict__ w1, const T *__restrict__ w2, const int32_t *__restrict__ sorted_pair,
                   const int32_t *__restrict__ tile_expert, const int32_t *__restrict__ counters, int top, int K, int N, int act, float limit, float slope,
                   int gather, T *__restrict__ inter, float *__restrict__ pair_out) {
    if ((int)blockIdx.x >= counters[0]) return;
    __shared__ float sa[kBK][kTileRows + 1];
    __shared__ float sb1[kBK][kBN + 1];
    __shared__ float sb2[GATED ? kBK : 1][kBN + 1];
    __shared__ int src_row[kTileRows];
    const int e = tile_expert[blockIdx.x];
    const int row0 = blockIdx.x * kTileRows, col0 = blockIdx.y * kBN;
    if (threadIdx.x < kTileRows) {
        // the first product gathers rows of h (or of its scaled copy); the second reads the sorted intermediate rows
        src_row[threadIdx.x] = moe_src_row(sorted_pair[row0 + threadIdx.x], row0 + (int)threadIdx.x, top, gather);
    }
    __syncthreads();
    const T *wa = w1 + (size_t)e * N * K;
    const T *wb = GATED ? w2 + (size_t)e * N * K : nullptr;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
    float c1[2][4] = {}, c2[2][4] = {};
    for (int k0 = 0; k0 < K; k0 += kBK) {
        for (int i = threadIdx.x; i < kTileRows * kBK; i += 256) {
            int r = i / kBK, k = i % kBK;
            int sr = src_row[r];
            sa[k][r] = (sr >= 0 && k0 + k < K) ? to_f(a[(size_t)sr * K + k0 + k]) : 0.f;
        }
        for (int i = threadIdx.x; i < kBN * kBK; i += 256) {
            int n = i / kBK, k = i % kBK;
            bool ok = col0 + n < N && k0 + k < K;
            sb1[k][n] = ok ? to_f(wa[(size_t)(col0 + n) * K + k0 + k]) : 0.f;
            if (GATED) sb2[k][n] = ok ? to_f(wb[(size_t)(col0 + n) * K + k0 + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kBK; ++k) {
            float a0 = sa[k][2 * ty], a1 = sa[k][2 * ty + 1];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float b = sb1[k][tx + 16 * c];
                c1[0][c] = fmaf(a0, b, c1[0][c]);
                c1[1][c] = fmaf(a1, b, c1[1][c]);
                if (GATED) {
                    float b2 = sb2[k][tx + 16 * c];
                    c2[0][c] = fmaf(a0, b2, c2[0][c]);
                    c2[1][c] = fmaf(a1, b2, c2[1][c]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        int row = row0 + 2 * ty + r;
        int pair = sorted_pair[row];
        if (pair < 0) continue;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            int col = col0 + tx + 16 * c;
            if (col >= N) continue;
            if (GATED) inter[(size_t)row * N + col] = from_f<T>(gated_pair(c1[r][c], c2[r][c], act, limit, slope));
            else if (inter) inter[(size_t)row * N + col] = from_f<T>(moe_act(c1[r][c], act));
            else pair_out[(size_t)pair * N + col] = c1[r][c];
        }
    }
}

// out[pair, :] = gate[pair] * h[pair / top, :] rounded to T: the rows of experts whose weight multiplies their input.
template <typename T>
__global__ void moe_scale_rows_kernel(const T *__restrict__ h, const float *__restrict__ gate, T *__restrict__ out, int top, int dim) {
    const int pair = blockIdx.x;
    const float g = gate[pair];
    const T *src = h + (size_t)(pair / top) * dim;
    for (int d = threadIdx.x; d < dim; d += blockDim.x) out[(size_t)pair * dim + d] = from_f<T>(g * to_f(src[d]));
}

// idx != NULL: a choice whose expert id is >= experts is an identity expert, its output the token's input row h[t, :].  A thread
// sums W columns; W = 4: a CTA takes 1024 columns of a token and all its choices' rows are on their way at once (2048 tokens of 6
// choices and 2048 columns: 37 -> 22 us, 16 tokens: 13 -> 3 us; before, a column and a choice at a time).
template <typename T, int W>
__global__ void __launch_bounds__(256)
moe_combine_kernel(const float *pair_out, const float *gate, const T *shared, const float *shared_gate, const int32_t *idx, int experts, const T *h, float *__restrict__ y,
                   int top, int dim) {
    const int t = blockIdx.x, d = (blockIdx.y * 256 + threadIdx.x) * W;
    tl::griddep_wait();  // all operands may be the launch before's: read by ld_cg, which stays behind it
    if (d >= dim) return;
    constexpr int AT_ONCE = 8;
    float s[W] = {};
    T beside[W];
    float beside_gate = 1.f;
    if (shared) {
        if (shared_gate) beside_gate = tl::ld_cg(shared_gate + t);
#pragma unroll
        for (int j = 0; j < W; ++j) beside[j] = tl::ld_cg(shared + (size_t)t * dim + d + j);
    }
    for (int k0 = 0; k0 < top; k0 += AT_ONCE) {
        float x[AT_ONCE][W], g[AT_ONCE];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u)
            if (k0 + u < top) {
                const size_t pair = (size_t)t * top + k0 + u;
                g[u] = gate ? tl::ld_cg(gate + pair) : 1.f;
                if (idx != nullptr && tl::ld_cg(idx + pair) >= experts) {
#pragma unroll
                    for (int j = 0; j < W; ++j) x[u][j] = to_f(tl::ld_cg(h + (size_t)t * dim + d + j));
                } else if constexpr (W == 4) {
                    const uint4 v = tl::ld_cg(reinterpret_cast<const uint4 *>(pair_out + pair * dim + d));
                    x[u][0] = __uint_as_float(v.x), x[u][1] = __uint_as_float(v.y), x[u][2] = __uint_as_float(v.z), x[u][3] = __uint_as_float(v.w);
                } else {
                    static_assert(W == 1, "columns of a thread");
                    x[u][0] = tl::ld_cg(pair_out + pair * dim + d);
                }
            }
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u)
            if (k0 + u < top) {
#pragma unroll
                for (int j = 0; j < W; ++j) s[j] = fmaf(g[u], x[u][j], s[j]);
            }
    }
    if (shared) {
#pragma unroll
        for (int j = 0; j < W; ++j) s[j] = fmaf(beside_gate, to_f(beside[j]), s[j]);
    }
    if constexpr (W == 4) *reinterpret_cast<float4 *>(y + (size_t)t * dim + d) = make_float4(s[0], s[1], s[2], s[3]);
    else y[(size_t)t * dim + d] = s[0];
}

}  // namespace tlb

using namespace tlb;

static int moe_product(const char *what, const MoeProduct &p, int dtype, cudaStream_t st) {
    if (moe_tc_ok(dtype, p.K, p.x, p.w0, p.w1)) {
        if (int e = moe_tc_product(p, st)) return e;
    } else {
        const dim3 grid((unsigned)(tlb_moe_max_rows(p.tokens, p.top, p.experts) / kTileRows), ceil_div(p.N, kBN));
        const MoeLists &l = p.lists;
        if (p.w1)
            TLB_DISPATCH(dtype, what, moe_grouped_kernel<T, true><<<grid, 256, 0, st>>>((const T *)p.x, (const T *)p.w0, (const T *)p.w1, l.sorted_pair, l.tile_expert,
                                                                                        l.counters, p.top, p.K, p.N, p.act, p.limit, p.slope, p.gather, (T *)p.inter, p.pair_out));
        else
            TLB_DISPATCH(dtype, what, moe_grouped_kernel<T, false><<<grid, 256, 0, st>>>((const T *)p.x, (const T *)p.w0, nullptr, l.sorted_pair, l.tile_expert,
                                                                                         l.counters, p.top, p.K, p.N, p.act, p.limit, p.slope, p.gather, (T *)p.inter, p.pair_out));
    }
    TL_LAUNCH_CHECK(what);
    return TL_OK;
}

extern "C" {

int tlb_moe_route(const void *h, const void *w, const void *b, int tokens, int dim, int experts, int top, int scoring, const void *choice_bias,
                  float weight_scale, int group_count, int group_keep, const void *aux_w, float *aux, int32_t *idx, float *gate, int dtype, void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!h || !w || !idx || !gate || dim <= 0 || experts <= 0 || top <= 0 || top > experts || scoring < 0 || scoring > 2)
        return tl::fail(TL_EINVAL, "moe_route: bad argument");
    if ((aux_w == nullptr) != (aux == nullptr) || group_count < 0 || group_keep < 0 || group_keep > group_count ||
        (group_count > 0 && (experts % group_count || group_keep * (experts / group_count) < top)))
        return tl::fail(TL_EINVAL, "moe_route: bad groups or side output");
    const size_t es = dtype == TL_BF16 ? 2 : 4;
    const auto bytes = [&](int tok) { return (((size_t)tok * dim * (tok == 1 ? es : sizeof(float)) + 15) & ~(size_t)15) + (size_t)tok * (2 * (size_t)experts + group_count) * sizeof(float); };
    if (bytes(1) > 48 * 1024) return tl::fail(TL_EINVAL, "moe_route: width %d + %d experts do not fit", dim, experts);
    const bool wide = dim * es % 16 == 0 && tl::aligned16(h) && tl::aligned16(w) && (!aux_w || tl::aligned16(aux_w));
    // eight tokens a CTA as long as a CTA's share of shared memory allows it; few tokens: a CTA each with more warps, so that no warp walks many rows of
    // weights (64 x 2048: 256 tokens a CTA each 11 us, eight a CTA 18; 400 20 and 19; 1024 39 and 19; 2048 68 and 27)
    const bool many = tokens >= 400 && bytes(8) <= 227 * 1024;
    const bool few = experts + (aux_w ? 1 : 0) <= 16;  // two rows a warp are all there are
    const int threads = many || tokens > 148 ? 256 : 512;
    const auto ready = [&](auto kernel, int tok) -> int {
        // on every call, because the attribute belongs to the device that is current
        if (bytes(tok) > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
            cudaGetLastError();
            return tl::fail(TL_ECUDA, "moe_route: no shared memory");
        }
        return TL_OK;
    };
#define TLB_ROUTE(TOK, ROWS, WV)                                                                                                                         \
    do {                                                                                                                                            \
        if (int e = ready(moe_route_kernel<T, TOK, ROWS, WV>, TOK)) return e;                                                                             \
        moe_route_kernel<T, TOK, ROWS, WV><<<ceil_div(tokens, TOK), threads, bytes(TOK), as_stream(stream)>>>(                                            \
            (const T *)h, (const T *)w, (const T *)b, tokens, dim, experts, top, scoring, (const T *)choice_bias, weight_scale, group_count,         \
            group_keep, (const T *)aux_w, aux, idx, gate);                                                                                           \
    } while (0)
    TLB_DISPATCH(dtype, "moe_route",
                 if (wide && many) { if (few) TLB_ROUTE(8, 2, (16 / (int)sizeof(T))); else TLB_ROUTE(8, 4, (16 / (int)sizeof(T))); }
                 else if (wide) TLB_ROUTE(1, 4, (16 / (int)sizeof(T)));
                 else { if (many) TLB_ROUTE(8, 4, 1); else TLB_ROUTE(1, 4, 1); });
#undef TLB_ROUTE
    TL_LAUNCH_CHECK("moe_route");
    return TL_OK;
}

int tlb_moe_gate_up(const void *h, const void *wg, const void *wu, int32_t *lists, int tokens, int top, int experts, int dim, int ff, int act, float limit,
                    float slope, void *inter, int dtype, void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!h || !wg || !wu || !lists || !inter || experts <= 0 || dim <= 0 || ff <= 0 || top <= 0 || (act != 0 && act != 1 && act != 3) || (act == 3 && !(limit > 0.f)))
        return tl::fail(TL_EINVAL, "moe_gate_up: bad argument");
    return moe_product("moe_gate_up", {h, wg, wu, moe_lists(lists, tokens, top, experts), tokens, top, experts, dim, ff, act, kGatherToken, limit, slope, inter, nullptr}, dtype,
                       as_stream(stream));
}

// The first product of experts without a gate: inter[row, :] = act(W[e] a[src(row)]), a = token rows (rows_are_pairs = 0) or one row per
// (token, choice) pair (rows_are_pairs = 1: the scaled copies tlb_moe_scale_rows makes).
int tlb_moe_up(const void *a, const void *wu, int32_t *lists, int tokens, int top, int experts, int dim, int ff, int act, int rows_are_pairs, void *inter, int dtype,
               void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!a || !wu || !lists || !inter || experts <= 0 || dim <= 0 || ff <= 0 || top <= 0 || act < 0 || act > 2) return tl::fail(TL_EINVAL, "moe_up: bad argument");
    return moe_product("moe_up", {a, wu, nullptr, moe_lists(lists, tokens, top, experts), tokens, top, experts, dim, ff, act, rows_are_pairs ? kGatherPair : kGatherToken, 0.f,
                                  1.f, inter, nullptr}, dtype, as_stream(stream));
}

int tlb_moe_scale_rows(const void *h, const float *gate, void *out, int tokens, int top, int dim, int dtype, void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!h || !gate || !out || top <= 0 || dim <= 0) return tl::fail(TL_EINVAL, "moe_scale_rows: bad argument");
    TLB_DISPATCH(dtype, "moe_scale_rows",
                 moe_scale_rows_kernel<T><<<tokens * top, 128, 0, as_stream(stream)>>>((const T *)h, gate, (T *)out, top, dim));
    TL_LAUNCH_CHECK("moe_scale_rows");
    return TL_OK;
}

static int moe_down(const void *inter, const void *wd, int32_t *lists, int tokens, int top, int experts, int dim, int ff, float *pair_out, int dtype, void *stream,
                    bool second) {
    if (tokens <= 0) return TL_OK;
    if (!inter || !wd || !lists || !pair_out || experts <= 0 || dim <= 0 || ff <= 0 || top <= 0) return tl::fail(TL_EINVAL, "moe_down: bad argument");
    return moe_product("moe_down", {inter, wd, nullptr, moe_lists(lists, tokens, top, experts), tokens, top, experts, ff, dim, 0, kGatherSorted, 0.f, 1.f, nullptr, pair_out, second},
                       dtype, as_stream(stream));
}
int tlb_moe_down(const void *inter, const void *wd, int32_t *lists, int tokens, int top, int experts, int dim, int ff, float *pair_out, int dtype, void *stream) {
    return moe_down(inter, wd, lists, tokens, top, experts, dim, ff, pair_out, dtype, stream, false);
}
int tlb_moe_down_next(const void *inter, const void *wd, int32_t *lists, int tokens, int top, int experts, int dim, int ff, float *pair_out, int dtype, void *stream) {
    return moe_down(inter, wd, lists, tokens, top, experts, dim, ff, pair_out, dtype, stream, true);
}

int tlb_moe_combine(const float *pair_out, const float *gate, const void *shared, const float *shared_gate, const int32_t *idx, int experts, const void *h, float *y, int tokens,
                    int top, int dim, int dtype, void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!pair_out || !y || top <= 0 || dim <= 0 || (idx && !h)) return tl::fail(TL_EINVAL, "moe_combine: bad argument");
    const bool wide = dim % 4 == 0 && tl::aligned16(pair_out) && tl::aligned16(y);
    const dim3 grid(tokens, ceil_div(dim, wide ? 1024 : 256));
#define TLB_COMBINE(WV) moe_launch(moe_combine_kernel<T, WV>, grid, 256, 0, as_stream(stream), pair_out, gate, (const T *)shared, shared_gate, idx, experts, (const T *)h, y, top, dim)
    TLB_DISPATCH(dtype, "moe_combine", if (wide) TLB_COMBINE(4); else TLB_COMBINE(1));
#undef TLB_COMBINE
    TL_LAUNCH_CHECK("moe_combine");
    return TL_OK;
}

}  // extern "C"
