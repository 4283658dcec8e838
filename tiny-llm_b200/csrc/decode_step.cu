// One decoding step of a Qwen3 model as ONE launch, for a few requests: embedding, all blocks, norm, head and greedy argmax
// (src/tiny_llm_ref/qwen3_week3.py:55-121,139-146,196-207,320-338 at L == 1), every rounding point of the operator sequence kept.
//
// What bounds a step of one request is not its bytes but its chain: a block is four products and an attention, each
// needs all of the one before, and each moves 5 to 28 MB, 1 to 4 us.  As a chain of launches (six a block: w4a16_matvec.cu, decode_attention_fused.cu)
// a link took 9 us, of which the fill of the pipeline, the hand-over to the next launch and the staging behind it were more than half.
// Here one CTA an SM lives for the whole step (a cooperative launch: the CTAs wait on one another) and a link costs one trip through L2:
//
//   * a producer stores its outputs as 8-byte packets, two bf16 values (or one float) and a 32-bit tag; a consumer reads the packets it needs
//     until they carry the step's tag.  An 8-byte store is seen whole or not at all, so the tag says that its values are there: no fence, no
//     counter, no barrier between the CTAs, and the wait IS the load of the activations;
//   * the weights do not depend on anything: every warp has a ring of four units (139 KB an SM) that runs ahead over the products' borders, so HBM works
//     through the exchange, the norm and the attention.  They lie in memory in the order in which the lanes hold them (decode_step_pack_kernel), so a
//     bulk copy brings two of them, scales and biases included, and a warp reads them without a bank conflict;
//   * an attention's older keys and values are requested before the activations of its q|k|v are waited for;
//   * the residual of a CTA's own rows never leaves its shared memory (o and down deal their rows to the same CTAs).
//
// Measured (eight Qwen3-4B blocks and the head, context 1011, a graph of the step alone): 483 us as 53 launches, 277 us here; 0.6B at 500: 315 -> 181.
// A key of the longest share of an attention costs 49 ns a block, 4 to 15 in the chain, so long contexts belong to the chain (the engine's rule, with the figures): 4B, four
// requests of 1000 tokens 485 us here and 660 there, of 8000 1170 and 871; one of 8000 440 and 612, of 32000 944 and 764.  What it went through (the same case): weights in registers
// across the phases 398; units in the lanes' order by bulk copies 348; digits on the integer tensor cores (ds_digits) 319; two units a copy
// and a barrier 303; sums by a thread an output instead of a half-warp, the norms' weights asked into L2 a block ahead 277.
// A block takes 28 us where its bytes take 8.  Counters (two blocks and the head, 105 us under the profiler): issue slots 41 % busy, DRAM 38 %, tensor pipe 8 %;
// of the 9.6 cycles between two instructions of a warp 2.4 wait for memory (packets, mostly), 1.8 at barriers, 1.5 for the instruction before.
//
// Rows are dealt in pieces of 8 or 16.  For 2560 rows over 148 CTAs 16 is too coarse (two pieces in some CTAs where the mean is 1.08), so o, down and q|k|v
// use pieces of 8: the M side of the MMA takes the 8 rows' first half of the reduction as its rows 0-7 and the second half as rows 8-15, and
// columns 0-3 / 4-7 of the N side hold the (up to four) tokens' activations of the two halves; the other two quarters of the
// result are not used.  That is why it ends at four tokens.
//
// Packets are reused every second block.  A CTA writes block l + 2's packets of a product only after it has received
// block l + 1's sums, to which every CTA contributed behind its own reads of block l: all CTAs own rows of gate|up (the launch refuses sizes where one would not).
// Tags never repeat between two writes of a place: step number x (blocks + 1) + block + 2, the embedding's one less.  None is 0, which the
// zeroed memory of a fresh workspace carries.
//
// A wait is bounded: one that runs out marks its CTA, whose further waits end soon.  Who gives up takes NaN for what did not come: packets, a unit's scales,
// an attention's scores.  So every sum that needed it is NaN, the next norm makes everybody's rows NaN, and nothing checks the mark on the way (a read of it before the
// stores took 3 % of the step).  The CTA's logits are NaN, the step's tokens -1, and the kernel's count of given-up waits goes up.
#include <limits.h>
#include <math_constants.h>

#include "common.cuh"
#include "kernels.h"
#include "per_device.h"
#include "tc_wait.cuh"
#include "w4a16_item.cuh"

namespace tl {

namespace {

typedef __nv_bfloat16 bf16;
constexpr int DS_WARPS = 16;
constexpr int DS_THREADS = DS_WARPS * 32;
constexpr int DS_UNIT = 4 * 512 + 128;       // bytes of a weight unit: four 16-byte words a lane; per g = 0..7 the scales of rows g, g + 8 and their biases (two groups a word)
constexpr int DS_MAX_LAYERS = 96;           // 11 KB of kernel parameters
constexpr int DS_HEAD = 128;                // head size
constexpr int DS_KV_STRIDE = 528;           // bytes of a staged token: K row | V row | 16 bytes that spread the banks
constexpr int DS_PART = 132;                // packets of a split's partial result of one head: 128 values, maximum, sum, 2 unused
constexpr int DS_SPLIT_TOKENS = 64;         // a key range is cut no finer than this
constexpr int DS_MAX_PIECES = 64;           // of a CTA and a product of a block
constexpr int DS_MAX_SPLITS = 32;           // one lane per split in the merge
constexpr float DS_LOG2E = 1.44269504089f;
constexpr float DS_NEG = -1e30f;
constexpr int DS_POLLS = 1 << 20;           // about half a second
constexpr uint32_t DS_NAN2 = 0x7fff7fffu;   // two bf16

struct DsMat {
    const uint32_t *w;
    const void *s, *b;
};
struct DsLayer {
    const unsigned char *w[4];  // q|k|v, o, gate|up, down, as units
    const bf16 *ln1, *ln2, *q_norm, *k_norm;
    bf16 *k_pages, *v_pages;
    const int32_t *table;
    int num_pages;
    float ln1_eps, ln2_eps, q_eps, k_eps, scale;
};
struct DsArgs {
    int layers, M, Hq, Hkv, D, ff, V;
    int page_size, max_pages, nsplit, kv_tokens, own_rows;
    unsigned int page_inverse;  // ceil(2^32 / page_size): x / page_size is the high word of x * page_inverse while x * page_size < 2^32
    float norm_eps;
    int act_off, act_bytes, asum_bytes, entry_bytes, kv_off;  // shared memory: pieces
    const int32_t *tokens, *offsets, *context_lens;
    const double *inv_freq;
    DsMat emb;
    const unsigned char *head;
    const bf16 *norm;
    bf16 *logits;
    int32_t *next_tokens;
    unsigned int *seq;                  // step number, limit of a wait's polls (0: DS_POLLS)
    unsigned char *best;                // [grid][M] 16 bytes
    unsigned char *xchg[2];             // packets of even and odd blocks
    unsigned int o_y, o_xo, o_act, o_xd, o_part;  // byte offsets in xchg[.] (q|k|v first)
    DsLayer layer[DS_MAX_LAYERS];
};

__device__ __forceinline__ float ds_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ ulonglong2 ds_ld2(const void *p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ds_ld(const void *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ds_st(void *p, uint32_t data, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((static_cast<unsigned long long>(tag) << 32) | data) : "memory");
}
__device__ __forceinline__ uint32_t ds_tag(unsigned long long v) { return static_cast<uint32_t>(v >> 32); }

// A failed poll: false when the wait is over for good.  dead: whether the CTA is marked, and the limit.
__device__ __forceinline__ bool ds_again(uint32_t &spins, volatile int *dead) {
    if ((++spins & 63u) != 0) return true;
    if (spins > static_cast<uint32_t>(dead[1])) *dead = 1;
    return *dead == 0;
}
__device__ __forceinline__ unsigned long long ds_poll(const void *p, uint32_t tag, volatile int *dead) {
    unsigned long long v = ds_ld(p);
    for (uint32_t spins = 0; ds_tag(v) != tag && ds_again(spins, dead);) v = ds_ld(p);
    return v;
}
// Whole warps: until the phase is over (true) or the wait is.
__device__ __forceinline__ bool ds_wait(uint32_t bar, uint32_t parity, volatile int *dead) {
    uint32_t done, spins = 0;
    bool over;
    do {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        over = __all_sync(0xffffffffu, done);
    } while (!over && ((spins & 63u) != 63u ? (++spins, true) : __all_sync(0xffffffffu, ds_again(spins, dead))));
    __syncwarp();
    return over;
}
__device__ __forceinline__ float ds_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void ds_ldmatrix(uint32_t (&r)[4], uint32_t p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(p) : "memory");
}

__device__ __forceinline__ void ds_cp16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 ds_lds(uint32_t p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p) : "memory");
    return v;
}

// Eight entries of an embedding row: value = float(code) * scale + bias, rounded once; rows outside the table are zero.
__device__ __forceinline__ uint4 ds_embed(const DsMat &e, int token, int V, int D, int c) {
    if (token < 0 || token >= V) return make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w = e.w[static_cast<size_t>(token) * (D / 8) + c];
    const size_t g = static_cast<size_t>(token) * (D / 128) + c / 16;
    const float s = __bfloat162float(static_cast<const bf16 *>(e.s)[g]), b = __bfloat162float(static_cast<const bf16 *>(e.b)[g]);
    auto v = [&](int i) { return static_cast<float>((w >> (4 * i)) & 0xFu) * s + b; };
    return make_uint4(pack2<bf16>(v(0), v(1)), pack2<bf16>(v(2), v(3)), pack2<bf16>(v(4), v(5)), pack2<bf16>(v(6), v(7)));
}

// One token: activations as integers.  The codes of a weight word are whole bytes after one mask (codes 0, 2, 4, 6) or a shift and a mask (1, 3, 5, 7), where bf16
// operands take seven operations a word, and those bound the consumer (ALU pipe: two cycles an operation).  So the tensor cores multiply
// unsigned codes by signed digits: an activation is d0 2^16 + d1 2^8 + d2 in units of 2^-21 of the power of two at or below its group's largest, the
// three digits are three columns of the N side, and their sums are exact.
// As an operand that is fewer bits than bf16 for small values: those down to 2^-14 of the group's largest are held exactly, smaller ones rounded to that unit, and
// below 2^-22 they are 0.  In return no sum is rounded, where the bf16 form takes 128 + code times the activations out of fp32 sums again, which loses as much: error of
// the logits against 64 bits, 48 inputs of one request (4B, eight blocks, contexts 300 and 1011), digits / bf16 operands 1.0002 +- 0.0013 (one input: 0.982 to
// 1.019), digits / chain of launches 1.0003 +- 0.0012.
// The 16 lanes of a half-warp hold one group of 128.  p0..p2: where this lane's 8 digits go; factors: where the columns' factors and sums go (first lane of the group).
__device__ __forceinline__ void ds_digits(uint4 raw, bool in, uint2 *p0, uint2 *p1, uint2 *p2, float *factors, float sum) {
    auto larger = [](uint32_t p, uint32_t q) {
        uint32_t r;
        asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(q));
        return r;
    };
    const uint32_t sign = 0x7fff7fffu;
    uint32_t pair = larger(larger(raw.x & sign, raw.y & sign), larger(raw.z & sign, raw.w & sign));
#pragma unroll
    for (int k = 8; k > 0; k >>= 1) pair = larger(pair, __shfl_xor_sync(0xffffffffu, pair, k));
    const uint32_t top = max(pair << 16, pair & 0xffff0000u);  // the largest magnitude's bits: of infinities and NaN the exponent is all ones
    const float2 f0 = unpack2<bf16>(raw.x), f1 = unpack2<bf16>(raw.y), f2 = unpack2<bf16>(raw.z), f3 = unpack2<bf16>(raw.w);
    const float f[8] = {f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y};
    const int e = static_cast<int>(top >> 23);
    const int field = min(275 - e, 254);  // exponent of the factor 2^(21 - floor(log2 top))
    const float up = __uint_as_float(static_cast<uint32_t>(field) << 23);
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = (__float_as_uint(fmaf(f[i], up, 12582912.f)) - 0x4B400000u + 0x00808080u) ^ 0x00808080u;  // rounded to an integer; three balanced digits, a byte each
    if (!in) return;
    // the bytes of four words at a time, transposed: digits of codes 0, 2, 4, 6 and of 1, 3, 5, 7
    uint32_t t[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t lo = __byte_perm(w[k], w[k + 2], 0x5140), hi = __byte_perm(w[k + 4], w[k + 6], 0x5140);
        t[k][2] = __byte_perm(lo, hi, 0x5410), t[k][1] = __byte_perm(lo, hi, 0x7632);
        t[k][0] = __byte_perm(__byte_perm(w[k], w[k + 2], 0x62), __byte_perm(w[k + 4], w[k + 6], 0x62), 0x5410);
    }
    *p0 = make_uint2(t[0][0], t[1][0]), *p1 = make_uint2(t[0][1], t[1][1]), *p2 = make_uint2(t[0][2], t[1][2]);
    if (factors != nullptr) {
        const float down = e == 255 ? __uint_as_float(0x7fffffffu) : field == 254 ? __uint_as_float(0x00400000u) : __uint_as_float(static_cast<uint32_t>(254 - field) << 23);
        reinterpret_cast<float4 *>(factors)[0] = make_float4(down * 65536.f, down * 256.f, sum, 0.f);  // columns 0 and 1, 2 and 3
        reinterpret_cast<float4 *>(factors)[1] = make_float4(down, 0.f, 0.f, 0.f);
    }
}

// acc += dequantised (16 rows x 2 groups) . digits, columns 2t, 2t + 1 of this lane.  unit: this lane's words, sb: its rows' scales and biases, digits: its columns'
// digits (512 bytes a group), factors: {factor, factor, sum, sum} of its columns (32 bytes a group).
// (Plain loads and no volatile assembly here: the compiler overlaps a group's loads with the products of the one before.)
__device__ __forceinline__ void ds_consume_digits(const unsigned char *unit, const unsigned char *sb, const unsigned char *digits, const unsigned char *factors, float (&acc)[4]) {
    const uint4 sbw = *reinterpret_cast<const uint4 *>(sb);
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const uint4 w0 = *reinterpret_cast<const uint4 *>(unit + it * 1024), w8 = *reinterpret_cast<const uint4 *>(unit + it * 1024 + 512);
        const float4 f = *reinterpret_cast<const float4 *>(factors + it * 32);
        const uint32_t x0[4] = {w0.x, w0.y, w0.z, w0.w}, x8[4] = {w8.x, w8.y, w8.z, w8.w};
        uint32_t d[4] = {0x4B400000u, 0x4B400000u, 0x4B400000u, 0x4B400000u};  // the sums (below 2^18) in the mantissa of 1.5 * 2^23
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint2 b = *reinterpret_cast<const uint2 *>(digits + (it * 4 + j) * 128);
            asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                         : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                         : "r"(x0[j] & 0x0F0F0F0Fu), "r"(x8[j] & 0x0F0F0F0Fu), "r"((x0[j] >> 4) & 0x0F0F0F0Fu), "r"((x8[j] >> 4) & 0x0F0F0F0Fu), "r"(b.x), "r"(b.y));
        }
        const float s0 = it == 0 ? W4Num<bf16>::lo(sbw.x) : W4Num<bf16>::hi(sbw.x), s8 = it == 0 ? W4Num<bf16>::lo(sbw.y) : W4Num<bf16>::hi(sbw.y);
        const float b0 = it == 0 ? W4Num<bf16>::lo(sbw.z) : W4Num<bf16>::hi(sbw.z), b8 = it == 0 ? W4Num<bf16>::lo(sbw.w) : W4Num<bf16>::hi(sbw.w);
        acc[0] = fmaf(b0, f.z, fmaf(s0 * f.x, __uint_as_float(d[0]) - 12582912.f, acc[0]));
        acc[1] = fmaf(b0, f.w, fmaf(s0 * f.y, __uint_as_float(d[1]) - 12582912.f, acc[1]));
        acc[2] = fmaf(b8, f.z, fmaf(s8 * f.x, __uint_as_float(d[2]) - 12582912.f, acc[2]));
        acc[3] = fmaf(b8, f.w, fmaf(s8 * f.y, __uint_as_float(d[3]) - 12582912.f, acc[3]));
    }
}

// The same with bf16 operands (two to four tokens; the arithmetic of w4_consume in w4a16_item.cuh).
template <int MP>
__device__ __forceinline__ void ds_consume_bf16(const unsigned char *unit, const unsigned char *sb, const unsigned char *act, const unsigned char *asum, float (&acc)[4]) {
    const uint4 sbw = *reinterpret_cast<const uint4 *>(sb);
    auto mma = [](float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    };
    const uint32_t mask = k_w4_mask, magic = W4Num<bf16>::MAGIC;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const uint4 w0 = *reinterpret_cast<const uint4 *>(unit + it * 1024), w8 = *reinterpret_cast<const uint4 *>(unit + it * 1024 + 512);
        const uint32_t x0[4] = {w0.x, w0.y, w0.z, w0.w}, x8[4] = {w8.x, w8.y, w8.z, w8.w};
        const float2 sums = *reinterpret_cast<const float2 *>(asum + it * 32);
        const float a0 = sums.x, a1 = sums.y, c0 = a0 * W4Num<bf16>::NEG_OFFSET, c1 = a1 * W4Num<bf16>::NEG_OFFSET;
        float d[4] = {c0, c1, c0, c1};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 bf = *reinterpret_cast<const uint4 *>(act + (it * 4 + j) * MP * 64);
            const uint32_t p0 = w4_lop(x0[j], mask, magic), p1 = w4_lop(x0[j] >> 4, mask, magic), p2 = w4_lop(x0[j] >> 8, mask, magic), p3 = w4_lop(x0[j] >> 12, mask, magic);
            const uint32_t q0 = w4_lop(x8[j], mask, magic), q1 = w4_lop(x8[j] >> 4, mask, magic), q2 = w4_lop(x8[j] >> 8, mask, magic), q3 = w4_lop(x8[j] >> 12, mask, magic);
            mma(d, p0, q0, p1, q1, bf.x, bf.y);
            mma(d, p2, q2, p3, q3, bf.z, bf.w);
        }
        const float s0 = it == 0 ? W4Num<bf16>::lo(sbw.x) : W4Num<bf16>::hi(sbw.x), s8 = it == 0 ? W4Num<bf16>::lo(sbw.y) : W4Num<bf16>::hi(sbw.y);
        const float b0 = it == 0 ? W4Num<bf16>::lo(sbw.z) : W4Num<bf16>::hi(sbw.z), b8 = it == 0 ? W4Num<bf16>::lo(sbw.w) : W4Num<bf16>::hi(sbw.w);
        acc[0] = fmaf(b0, a0, fmaf(s0, d[0], acc[0]));
        acc[1] = fmaf(b0, a1, fmaf(s0, d[1], acc[1]));
        acc[2] = fmaf(b8, a0, fmaf(s8, d[2], acc[2]));
        acc[3] = fmaf(b8, a1, fmaf(s8, d[3], acc[3]));
    }
}

// The M rows of a product's activations, from their packets (layouts of act / asum: w4a16_item.cuh), normalised first where
// `norm` (the weights, in shared memory once every thread's copies have landed) is given.  The loads are repeated until the packets carry
// the tag.  With a norm a warp's 32 chunks of 8 are one row's (the host checks).  Ends with __syncthreads().
template <int MP>
__device__ __forceinline__ void ds_stage(const DsArgs &a, const unsigned char *src, uint32_t tag, const uint4 *norm, float eps, int N, uint4 *act,
                                         float *asum, float *sq, volatile int *dead) {
    constexpr int MPA = w4_mpa(MP);
    constexpr int FLIGHT = 3;  // chunks of a thread polled at a time
    const int words = N / 8, total = a.M * words;
    const int lane = threadIdx.x & 31;
    auto row_of = [&](int idx) {
        int m = 0;
#pragma unroll
        for (int i = 1; i < MP; ++i) m += idx >= i * words;
        return m;
    };
    auto place = [&](int m, int c) { return act + (((c >> 4) * 4 + (c & 3)) * MP + m) * 4 + ((c >> 2) & 3); };
    auto digit_place = [&](int c, int col) { return reinterpret_cast<uint2 *>(act) + (((c >> 4) * 4 + (c & 3)) * 4 + col) * 4 + ((c >> 2) & 3); };
    auto put = [&](int m, int c, uint4 v) {  // a chunk as it came: where its digits go, or where it stays
        if (MP == 1)
            *digit_place(c, 0) = make_uint2(v.x, v.y), *digit_place(c, 1) = make_uint2(v.z, v.w);
        else
            *place(m, c) = v;
    };
    auto get = [&](int m, int c) {
        if (MP != 1) return *place(m, c);
        const uint2 lo = *digit_place(c, 0), hi = *digit_place(c, 1);
        return make_uint4(lo.x, lo.y, hi.x, hi.y);
    };
    auto half_warp_sum = [](float v) {
#pragma unroll
        for (int k = 8; k > 0; k >>= 1) v += __shfl_xor_sync(0xffffffffu, v, k);
        return v;
    };
    bool lost = false;  // chunks of this thread did not come: all of its chunks are NaN below
#pragma unroll 1
    for (int base = threadIdx.x; base < total; base += DS_THREADS * FLIGHT) {
        const unsigned char *p = src + static_cast<size_t>(base) * 32;
        unsigned pending = 0;
#pragma unroll
        for (int j = 0; j < FLIGHT; ++j) pending |= base + j * DS_THREADS < total ? 1u << j : 0u;
        uint32_t spins = 0;
#pragma unroll 1
        while (pending != 0) {
            ulonglong2 v[FLIGHT][2];
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j)
                if (pending >> j & 1u) v[j][0] = ds_ld2(p + j * DS_THREADS * 32), v[j][1] = ds_ld2(p + j * DS_THREADS * 32 + 16);
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j)
                if ((pending >> j & 1u) && ds_tag(v[j][0].x) == tag && ds_tag(v[j][0].y) == tag && ds_tag(v[j][1].x) == tag && ds_tag(v[j][1].y) == tag) {
                    const int idx = base + j * DS_THREADS, m = row_of(idx);
                    put(m, idx - m * words, make_uint4(static_cast<uint32_t>(v[j][0].x), static_cast<uint32_t>(v[j][0].y), static_cast<uint32_t>(v[j][1].x), static_cast<uint32_t>(v[j][1].y)));
                    pending &= ~(1u << j);
                }
            if (pending != 0 && !ds_again(spins, dead)) {
                lost = true;
                break;
            }
        }
    }
    __syncwarp();
    if (norm != nullptr) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll 1
        for (int idx = threadIdx.x; idx < total; idx += DS_THREADS) {  // (this thread's own chunks)
            const int m = row_of(idx);
            const uint4 x = get(m, idx - m * words);
            const float2 f0 = unpack2<bf16>(x.x), f1 = unpack2<bf16>(x.y), f2 = unpack2<bf16>(x.z), f3 = unpack2<bf16>(x.w);
            const float part = half_warp_sum(f0.x * f0.x + f0.y * f0.y + f1.x * f1.x + f1.y * f1.y + f2.x * f2.x + f2.y * f2.y + f3.x * f3.x + f3.y * f3.y);
            if ((lane & 15) == 0) sq[idx >> 4] = part;  // 16 chunks a group: slot = row * N / 128 + group
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int idx = threadIdx.x; (idx & ~31) < total; idx += DS_THREADS) {
        const int m = row_of(idx), c = idx - m * words;
        const bool in = idx < total;
        uint4 raw = in ? get(m, c) : make_uint4(0u, 0u, 0u, 0u);
        if (norm != nullptr) {
            float ss = 0.f;
#pragma unroll 1
            for (int i = lane; i < N / 128; i += 32) ss += sq[m * (N / 128) + i];
            const float inv = rsqrtf(warp_sum(ss) / static_cast<float>(N) + eps);
            const uint4 w = norm[c];
            const float2 x0 = unpack2<bf16>(raw.x), x1 = unpack2<bf16>(raw.y), x2 = unpack2<bf16>(raw.z), x3 = unpack2<bf16>(raw.w);
            const float2 w0 = unpack2<bf16>(w.x), w1 = unpack2<bf16>(w.y), w2 = unpack2<bf16>(w.z), w3 = unpack2<bf16>(w.w);
            raw = make_uint4(pack2<bf16>(x0.x * inv * w0.x, x0.y * inv * w0.y), pack2<bf16>(x1.x * inv * w1.x, x1.y * inv * w1.y),
                             pack2<bf16>(x2.x * inv * w2.x, x2.y * inv * w2.y), pack2<bf16>(x3.x * inv * w3.x, x3.y * inv * w3.y));
        }
        if (lost) raw = make_uint4(DS_NAN2, DS_NAN2, DS_NAN2, DS_NAN2);
        const float2 f0 = unpack2<bf16>(raw.x), f1 = unpack2<bf16>(raw.y), f2 = unpack2<bf16>(raw.z), f3 = unpack2<bf16>(raw.w);
        const float part = half_warp_sum(((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y)));
        if (MP == 1) {
            ds_digits(raw, in, digit_place(c, 0), digit_place(c, 1), digit_place(c, 2), (c & 15) == 0 ? asum + (c >> 4) * 8 : nullptr, part);
        } else if (in) {  // element order [0,4,1,5,2,6,3,7], as w4_stage
            *place(m, c) = make_uint4(__byte_perm(raw.x, raw.z, 0x5410), __byte_perm(raw.x, raw.z, 0x7632), __byte_perm(raw.y, raw.w, 0x5410), __byte_perm(raw.y, raw.w, 0x7632));
            if ((c & 15) == 0) asum[(c >> 4) * MPA + m] = part;
        }
    }
    __syncthreads();
}

template <int MP, int BATCH, int BATCHES>
__global__ void __launch_bounds__(DS_THREADS, 1) decode_step_kernel(const __grid_constant__ DsArgs a) {
    constexpr int ENTRY = 16 * MP + 1;                 // floats of a (piece, warp) partial sum: 16 rows of the MMA, their tokens; odd, as a half-warp reads one value of 16 entries
    constexpr int Q_ROW = DS_HEAD + 8;                 // bf16 of a staged query head (the padding spreads the banks)
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int deals[5][4];                        // per kind of product: reduction, this CTA's first piece, its pieces, units of a piece
    __shared__ uchar2 span[4][DS_MAX_PIECES];          // the first and the last warp that have units of a piece
    __shared__ int4 shares[5][DS_WARPS];               // per kind and warp: first unit, one past the last, the first's piece and place in it
    __shared__ int dead_s[2];
    __shared__ __align__(8) unsigned long long kv_bar[2], full[DS_WARPS][BATCHES];
    __shared__ __align__(16) bf16 q_s[8 * Q_ROW], k_cur[DS_HEAD], v_cur[DS_HEAD];  // query heads (rows past the group stay zero); the newest key and value
    __shared__ float2 cs_s[DS_HEAD / 2];
    __shared__ float st_s[256];                        // per (head, tile of 8 tokens): maximum [4][32], sum [4][32]
    __shared__ float red_l[16];
    __shared__ float best_v[MP][DS_WARPS];
    __shared__ int best_i[MP][DS_WARPS];
    volatile int *dead = dead_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int cta = blockIdx.x, ctas = gridDim.x;
    const int M = MP == 1 ? 1 : a.M, D = a.D, Gq = a.Hq / a.Hkv;

    uint4 *act = reinterpret_cast<uint4 *>(smem + a.act_off);  // behind the warps' rings of weight units
    float *asum = reinterpret_cast<float *>(smem + a.act_off + a.act_bytes);
    float *sq = asum + a.asum_bytes / 4;
    float *entries = sq + a.asum_bytes / 4;
    uint4 *norm_s = reinterpret_cast<uint4 *>(entries + a.entry_bytes / 4);  // the next norm's weights
    float *own = reinterpret_cast<float *>(norm_s + D / 8);  // [M][own_rows] residual of this CTA's rows
    float *s_s = own + MP * a.own_rows;                // [4][kv_tokens] scores, then probabilities
    int *pg_s = reinterpret_cast<int *>(s_s + 4 * a.kv_tokens);  // page ids of a round
    const uint32_t kv_s = g_smem_u32(smem + a.kv_off);  // [kv_tokens][DS_KV_STRIDE], beside q|k|v's activations and under the wider ones
    float *red = entries;                              // the merge's weighted parts

    const int qkv_w = (a.Hq + 2 * a.Hkv) * DS_HEAD, q_w = a.Hq * DS_HEAD;
    const unsigned int epoch = *static_cast<volatile unsigned int *>(a.seq);
    const uint32_t tag0 = epoch * static_cast<uint32_t>(a.layers + 1) + 2u;

    // ---- this CTA's part of every attention: a request, a K/V head and a range of its keys
    const int item = cta / a.nsplit, split = cta - item * a.nsplit;
    const bool has_item = item < M * a.Hkv;
    const int ab = has_item ? item / a.Hkv : 0, kvh = has_item ? item - ab * a.Hkv : 0;
    const int ctx = min(a.context_lens[ab], a.max_pages * a.page_size);
    const int splits = max(1, min(a.nsplit, (ctx + DS_SPLIT_TOKENS - 1) / DS_SPLIT_TOKENS));
    const int per_split = ((max(ctx, 0) + splits - 1) / splits + 7) & ~7;
    const int k_begin = split * per_split, k_end = min(ctx, k_begin + per_split);
    const bool attends = has_item && split < splits, has_keys = attends && k_begin < k_end;
    const int cur_tok = ctx - 1;
    const int round = k_end - k_begin <= a.kv_tokens ? a.kv_tokens : a.kv_tokens / 2;  // one round, or rounds of half the space each, the next requested ahead
    const uint32_t by_splits = 65536u / splits + 1u;   // x / splits = x * by_splits >> 16 for x below 64
    auto page_of = [&](int tok) { return a.page_size == 1 ? tok : static_cast<int>(__umulhi(static_cast<uint32_t>(tok), a.page_inverse)); };

    // ---- products of the step: 4 * block + {0 q|k|v, 1 o, 2 gate|up, 3 down}, then the head.  The five kinds are dealt out alike in all blocks.
    const int products = 4 * a.layers;
    auto kind_of = [&](int s) { return s == products ? 4 : s & 3; };
    auto matrix = [&](int s) { return s == products ? a.head : a.layer[s >> 2].w[s & 3]; };
    for (int i = threadIdx.x; i < 8 * Q_ROW; i += DS_THREADS) q_s[i] = __ushort_as_bfloat16(0);
    if (threadIdx.x < 5 * DS_WARPS) {
        const int kind = threadIdx.x / DS_WARPS, w = threadIdx.x % DS_WARPS;
        const int rows = kind == 0 ? qkv_w : kind == 2 ? 2 * a.ff : kind == 4 ? a.V : D;
        const int N = kind == 1 ? q_w : kind == 3 ? a.ff : D;
        const bool half = kind != 2 && kind != 4;
        const unsigned all = static_cast<unsigned>(rows) >> (half ? 3 : 4);
        const int c0 = static_cast<int>(all * cta / ctas), pieces = static_cast<int>(all * (cta + 1) / ctas) - c0, P = N / (half ? 512 : 256);
        const int begin = pieces * P * w / DS_WARPS;
        shares[kind][w] = make_int4(begin, pieces * P * (w + 1) / DS_WARPS, begin / P, begin % P);
        if (kind < 4 && w == 0)
            for (int i = 0; i < pieces; ++i) {
                int first = DS_WARPS, last = 0;
                for (int v = 0; v < DS_WARPS; ++v) {
                    const int from = pieces * P * v / DS_WARPS, to = pieces * P * (v + 1) / DS_WARPS;
                    if (from < to && from < (i + 1) * P && to > i * P) first = min(first, v), last = v;
                }
                span[kind][i] = make_uchar2(first, last);
            }
        if (w == 0) deals[kind][0] = N, deals[kind][1] = c0, deals[kind][2] = pieces, deals[kind][3] = P;
    }
    if (threadIdx.x == 0) {
        const unsigned int limit = static_cast<volatile unsigned int *>(a.seq)[1];
        dead_s[0] = 0, dead_s[1] = limit == 0 ? DS_POLLS : static_cast<int>(min(limit, 1u << 30));
        g_mbar_init(g_smem_u32(&kv_bar[0]), DS_THREADS);
        g_mbar_init(g_smem_u32(&kv_bar[1]), DS_THREADS);
#pragma unroll 1
        for (int i = 0; i < DS_WARPS * BATCHES; ++i) g_mbar_init(g_smem_u32(&full[0][0] + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    // ---- a warp's units of all products, one after another, through its ring: BATCHES of up to BATCH units (one copy, one barrier) are in flight or
    // waiting to be used
    const uint32_t ring = g_smem_u32(smem) + warp * (BATCHES * BATCH * DS_UNIT), full0 = g_smem_u32(&full[warp][0]);
    const unsigned char *l_p = nullptr;  // next unit to request
    int l_left = 0, l_s = -1;
    auto request = [&](int slot) {
#pragma unroll 1
        while (l_left == 0 && l_s < products) {  // on to the next product
            l_s += 1;
            const int kind = kind_of(l_s);
            const int4 share = shares[kind][warp];
            l_left = share.y - share.x;
            l_p = matrix(l_s) + static_cast<size_t>(deals[kind][1] * deals[kind][3] + share.x) * DS_UNIT;
        }
        const int n = min(BATCH, l_left);
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %2;\n\t"
                     "@p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(ring + slot * (BATCH * DS_UNIT)), "l"(l_p),
                     "r"(n * DS_UNIT), "r"(full0 + slot * 8), "r"(lane == 0 ? n : 0)
                     : "memory");
        l_p += n * DS_UNIT;
        l_left -= n;
    };
    int u_slot = 0, u_parity = 0;
    // ---- keys and values of a round: its page ids and its rows, into buffer b (nothing reads it any more)
    auto request_keys = [&](const DsLayer &l, int rb, int b) {
        const int rend = min(k_end, rb + round), lp0 = page_of(rb), n = page_of(rend - 1) - lp0 + 1;
        const int32_t *const table = l.table + static_cast<size_t>(ab) * a.max_pages + lp0;
#pragma unroll 1
        for (int i = threadIdx.x; i < n; i += DS_THREADS) pg_s[b * (round + 4) + i] = table[i];
        const int c8 = lane & 15;
#pragma unroll 1
        for (int tok = rb + warp * 2 + (lane >> 4); tok < rend; tok += 2 * DS_WARPS) {
            const int lp = page_of(tok), pid = table[lp - lp0];
            if (tok != cur_tok && pid >= 0 && pid < l.num_pages) {
                const size_t off = (static_cast<size_t>(pid * a.Hkv + kvh) * a.page_size + (tok - lp * a.page_size)) * DS_HEAD + c8 * 8;
                const uint32_t dst = kv_s + (b * round + tok - rb) * DS_KV_STRIDE + c8 * 16;
                ds_cp16(dst, l.k_pages + off);
                ds_cp16(dst + 256, l.v_pages + off);
            }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(g_smem_u32(&kv_bar[b])) : "memory");
    };
    // What product s needs beside its weights: the norm's weights to shared memory (and those of the next block to L2), the attention's keys
    auto prepare = [&](int s) {
        const int kind = kind_of(s);
        if (kind == 0 || kind == 2 || kind == 4) {
            const bf16 *w = kind == 4 ? a.norm : kind == 0 ? a.layer[s >> 2].ln1 : a.layer[s >> 2].ln2;
#pragma unroll 1
            for (int c = threadIdx.x; c < D / 8; c += DS_THREADS) ds_cp16(g_smem_u32(norm_s + c), w + c * 8);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (kind == 0 && has_keys) request_keys(a.layer[s >> 2], k_begin, 0);
        if (kind == 1 && warp == DS_WARPS - 1 && cta < 8) {  // a read of these from HBM, behind the weights in flight, takes 2 us
            const bool last = (s >> 2) + 1 == a.layers;
            const DsLayer &next = a.layer[last ? 0 : (s >> 2) + 1];
            const int lines = D / 64;  // of 128 bytes
            for (int i = cta * 32 + lane; i < 2 * lines + 2; i += 8 * 32) {
                const bf16 *p = i < lines ? (last ? a.norm : next.ln1) + i * 64 : i < 2 * lines ? next.ln2 + (i - lines) * 64 : i == 2 * lines ? next.q_norm : next.k_norm;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
            }
        }
    };

#pragma unroll 1
    for (int k = 0; k < BATCHES; ++k) request(k);
    prepare(0);
    int kv_phase = 0;
    {  // the residual stream begins with the embedding: this CTA's rows, kept and handed round
        const int r0 = deals[1][1] * 8, rows = deals[1][2] * 8;
#pragma unroll 1
        for (int o = threadIdx.x; o < M * (rows / 8); o += DS_THREADS) {
            const int m = o / (rows / 8), r = (o - m * (rows / 8)) * 8;
            const uint4 e = ds_embed(a.emb, a.tokens[m], a.V, D, (r0 + r) / 8);
            const uint32_t w[4] = {e.x, e.y, e.z, e.w};
            for (int i = 0; i < 4; ++i) {
                own[m * a.own_rows + r + 2 * i] = W4Num<bf16>::lo(w[i]), own[m * a.own_rows + r + 2 * i + 1] = W4Num<bf16>::hi(w[i]);
                ds_st(a.xchg[1] + a.o_xd + (static_cast<size_t>(m) * (D / 2) + (r0 + r) / 2 + i) * 8, w[i], tag0 - 1u);
            }
        }
    }
    if (attends && threadIdx.x < DS_HEAD / 2) {  // a step's positions are the same in all blocks
        const float angle = static_cast<float>(static_cast<double>(a.offsets[ab]) * a.inv_freq[threadIdx.x]);
        float sn, cn;
        sincosf(angle, &sn, &cn);
        cs_s[threadIdx.x] = make_float2(cn, sn);
    }
    __syncthreads();

#pragma unroll 1
    for (int s = 0; s <= products; ++s) {
        const int kind = kind_of(s), li = s >> 2;
        const DsLayer &l = a.layer[kind == 4 ? a.layers - 1 : li];
        const uint32_t tag = tag0 + li;
        unsigned char *const x = a.xchg[li & 1];
        const bool half = kind != 2 && kind != 4;
        const int N = deals[kind][0], c0 = deals[kind][1], pieces = deals[kind][2], P = deals[kind][3];

        // ---- activations
        {
            const unsigned char *src = (kind == 0 || kind == 4) ? a.xchg[(li & 1) ^ 1] + a.o_xd : x + (kind == 1 ? a.o_y : kind == 2 ? a.o_xo : a.o_act);
            const uint4 *norm = kind == 1 || kind == 3 ? nullptr : norm_s;
            const float eps = kind == 4 ? a.norm_eps : kind == 0 ? l.ln1_eps : l.ln2_eps;
            ds_stage<MP>(a, src, kind == 0 || kind == 4 ? tag - 1u : tag, norm, eps, N, act, asum, sq, dead);
        }

        // ---- this warp's units
        {
            constexpr int GROUP = MP == 1 ? 512 : MP * 256;  // bytes of a staged group: four columns of digits, or bf16
            const unsigned char *act0 = reinterpret_cast<const unsigned char *>(act) + (MP == 1 ? (g & 3) * 32 + t * 8 : (g & (MP - 1)) * 64 + t * 16);
            const unsigned char *sums0 = reinterpret_cast<const unsigned char *>(asum) + (MP == 1 ? (t & 1) * 16 : (half ? t & 1 : t) * 8);
            if (half) act0 += g >= 4 ? P * 2 * GROUP : 0, sums0 += t >= 2 ? P * 2 * 32 : 0;  // columns 4-7 are the tokens at the second half of the reduction
            const int t8 = half ? t - 2 : t;  // lanes that hold the rows 8-15 of a token
            const int4 share = shares[kind][warp];
            const unsigned char *act_u = act0 + share.w * (2 * GROUP), *sums_u = sums0 + share.w * 64;
            int left = P - share.w;  // units of the piece
            float *e = entries + static_cast<size_t>(share.z + warp) * ENTRY + g * MP;
            if (share.x == share.y)  // no units (fewer of them than warps): nothing between its neighbours' shares of the piece
                for (int i = lane; i < ENTRY; i += 32) entries[static_cast<size_t>(share.z + warp) * ENTRY + i] = 0.f;
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int i = share.x; i < share.y; i += BATCH) {
                if (!ds_wait(full0 + u_slot * 8, u_parity, dead)) {  // the copy may still be in flight: the warp requests nothing more
                    l_left = 0, l_s = products;
                    for (int k = 0; k < BATCH; ++k) *reinterpret_cast<uint32_t *>(smem + ((warp * BATCHES + u_slot) * BATCH + k) * DS_UNIT + 2048 + lane * 4) = DS_NAN2;
                    __syncwarp();
                }
                const unsigned char *unit = smem + (warp * BATCHES + u_slot) * (BATCH * DS_UNIT);
                const int n = min(BATCH, share.y - i);
#pragma unroll 1
                for (int k = 0; k < n; ++k) {
                    if constexpr (MP == 1)
                        ds_consume_digits(unit + lane * 16, unit + 2048 + g * 16, act_u, sums_u, acc);
                    else
                        ds_consume_bf16<MP>(unit + lane * 16, unit + 2048 + g * 16, act_u, sums_u, acc);
                    unit += DS_UNIT, act_u += 2 * GROUP, sums_u += 64;
                    if (--left == 0 || i + k + 1 == share.y) {  // park the piece's sums
                        if (MP == 1) {  // the three digits' columns: two here, one in the next lane
                            acc[0] += acc[1] + __shfl_xor_sync(0xffffffffu, acc[0], 1);
                            acc[2] += acc[3] + __shfl_xor_sync(0xffffffffu, acc[2], 1);
                        }
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) {
                            if (2 * t + k2 < MP) e[2 * t + k2] = acc[k2];
                            if (t8 >= 0 && 2 * t8 + k2 < MP) e[8 * MP + 2 * t8 + k2] = acc[2 + k2];
                        }
                        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                        e += ENTRY, left = P, act_u = act0, sums_u = sums0;
                    }
                }
                __syncwarp();  // all lanes have read the batch
                request(u_slot);
                u_slot += 1;
                if (u_slot == BATCHES) u_slot = 0, u_parity ^= 1;
            }
        }
        __syncthreads();
        if (kind == 4) break;

        // ---- the pieces' sums, a thread an output: the shares of the few warps that had units of its piece, in warp order
        {
            const int shift = half || kind == 2 ? 3 : 4;  // outputs of a piece
            const int rows = pieces << shift, r0 = c0 << shift, outs = rows * M;
            unsigned char *const dst = x + (kind == 0 ? 0u : kind == 1 ? a.o_xo : kind == 2 ? a.o_act : a.o_xd);
            const int width = kind == 0 ? qkv_w : kind == 2 ? a.ff : D;
#pragma unroll 1
            for (int o = threadIdx.x; (o & ~31) < outs; o += DS_THREADS) {
                int m = 0, r = o;
#pragma unroll
                for (int i = 1; i < MP; ++i)
                    if (r >= rows) r -= rows, m += 1;
                float v = 0.f, v8 = 0.f;
                if (o < outs) {
                    const int piece = r >> 3, last = span[kind][piece].y;
                    int w = span[kind][piece].x;
                    const float *e = entries + static_cast<size_t>(piece + w) * ENTRY + (r & 7) * MP + m;
#pragma unroll 4
                    for (; w <= last; ++w, e += ENTRY) v += e[0], v8 += e[8 * MP];
                    if (kind == 2) {
                        const float gate = ds_round(v), up = ds_round(v8);
                        v = (gate / (1.0f + expf(-gate))) * up;
                    } else {
                        v += v8;  // the two halves of the reduction
                        if (kind != 0) {
                            float *const mine = own + m * a.own_rows + r;
                            v = ds_round(*mine + ds_round(v));
                            *mine = v;
                        }
                    }
                }
                const float next = __shfl_down_sync(0xffffffffu, v, 1);  // rows is even: a pair is one token's
                if (o < outs && (o & 1) == 0) ds_st(dst + (static_cast<size_t>(m) * (width / 2) + ((r0 + r) >> 1)) * 8, pack2<bf16>(v, next), tag);
            }
        }
        prepare(s + 1);

        // ---- attention, behind q|k|v
        if (kind == 0 && attends) {
            if (warp < Gq + 2) {  // this step's heads: norm and rotation, v as it is
                const bool is_q = warp < Gq, is_v = warp == Gq + 1;
                const int head = is_q ? kvh * Gq + warp : (is_v ? a.Hq + a.Hkv : a.Hq) + kvh;
                uint32_t w_lo = 0, w_hi = 0;
                if (!is_v) {
                    const uint32_t *w = reinterpret_cast<const uint32_t *>(is_q ? l.q_norm : l.k_norm);
                    w_lo = w[lane], w_hi = w[32 + lane];
                }
                const unsigned char *p = x + (static_cast<size_t>(ab) * (qkv_w / 2) + head * 64 + lane) * 8;
                unsigned long long lo = ds_ld(p), hi = ds_ld(p + 256);
#pragma unroll 1
                for (uint32_t spins = 0; ds_tag(lo) != tag || ds_tag(hi) != tag;) {
                    if (!ds_again(spins, dead)) {
                        lo = hi = DS_NAN2;
                        break;
                    }
                    lo = ds_ld(p), hi = ds_ld(p + 256);
                }
                __syncwarp();
                uint32_t o_lo = static_cast<uint32_t>(lo), o_hi = static_cast<uint32_t>(hi);
                if (!is_v) {
                    const float2 re = unpack2<bf16>(o_lo), im = unpack2<bf16>(o_hi);
                    const float inv = rsqrtf(warp_sum(re.x * re.x + im.x * im.x + re.y * re.y + im.y * im.y) / static_cast<float>(DS_HEAD) + (is_q ? l.q_eps : l.k_eps));
                    const float2 wr = unpack2<bf16>(w_lo), wi = unpack2<bf16>(w_hi);
                    const float2 cs0 = cs_s[2 * lane], cs1 = cs_s[2 * lane + 1];
                    const float r0n = ds_round(re.x * inv * wr.x), i0n = ds_round(im.x * inv * wi.x);
                    const float r1n = ds_round(re.y * inv * wr.y), i1n = ds_round(im.y * inv * wi.y);
                    o_lo = pack2<bf16>(r0n * cs0.x - i0n * cs0.y, r1n * cs1.x - i1n * cs1.y);
                    o_hi = pack2<bf16>(i0n * cs0.x + r0n * cs0.y, i1n * cs1.x + r1n * cs1.y);
                }
                uint32_t *const to = reinterpret_cast<uint32_t *>(is_q ? q_s + warp * Q_ROW : is_v ? v_cur : k_cur);
                to[lane] = o_lo;
                to[32 + lane] = o_hi;
            }
            // values: thread = (head oh, 8 columns d8, token sub of a tile); afterwards it keeps column sub of the eight
            const int oh = threadIdx.x >> 7, sub = threadIdx.x & 7, d8 = (threadIdx.x >> 3) & 15;
            float scale2 = l.scale * DS_LOG2E;
            float m_run = DS_NEG, l_run = 0.f, o_run = 0.f;
            if (!has_keys) __syncthreads();  // (each round begins with one) the sums of q|k|v have been read
#pragma unroll 1
            for (int rb = k_begin, b = 0; rb < k_end; rb += round, b ^= 1) {
                const int cnt = min(k_end - rb, round), lp0 = page_of(rb);
                const uint32_t kv_b = kv_s + b * round * DS_KV_STRIDE;
                const int *const pages = pg_s + b * (round + 4);
                if (rb != k_begin) __syncthreads();  // the last round's page ids, rows and scores are dead
                if (rb + round < k_end) request_keys(l, rb + round, b ^ 1);
                if (!ds_wait(g_smem_u32(&kv_bar[b]), kv_phase >> b & 1, dead)) scale2 = m_run = CUDART_NAN_F;
                kv_phase ^= 1 << b;
                __syncthreads();  // q_s / k_cur / v_cur and all copies of the round
                const int cur_slot = cur_tok - rb;
                if (cur_slot >= 0 && cur_slot < cnt) {  // the newest token joins the round and is appended to the cache
                    if (threadIdx.x < 2 * (DS_HEAD / 8)) {
                        const bool is_v = threadIdx.x >= DS_HEAD / 8;
                        const int ch = threadIdx.x & (DS_HEAD / 8 - 1);
                        const uint4 row = *reinterpret_cast<const uint4 *>((is_v ? v_cur : k_cur) + ch * 8);
                        *reinterpret_cast<uint4 *>(smem + a.kv_off + (b * round + cur_slot) * DS_KV_STRIDE + (is_v ? 256 : 0) + ch * 16) = row;
                        const int lp = page_of(cur_tok), pid = pages[lp - lp0];
                        if (pid >= 0 && pid < l.num_pages)
                            *reinterpret_cast<uint4 *>((is_v ? l.v_pages : l.k_pages) + (static_cast<size_t>(pid * a.Hkv + kvh) * a.page_size + (cur_tok - lp * a.page_size)) * DS_HEAD + ch * 8) = row;
                    }
                    __syncthreads();
                }
                // scores of 8 tokens x the heads of the group per MMA tile, with the tile's maximum and sum
#pragma unroll 1
                for (int tile = warp; tile * 8 < cnt; tile += DS_WARPS) {
                    float e[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                    const uint32_t krow = kv_b + (tile * 8 + (lane & 7)) * DS_KV_STRIDE + (lane >> 3) * 16;
                    const uint32_t qrow = g_smem_u32(q_s) + (lane & 7) * (Q_ROW * 2) + (lane >> 3) * 16;
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {  // 32 columns: both operands' fragments of two MMAs
                        uint32_t kf[4], qf[4];
                        ds_ldmatrix(kf, krow + ks * 64);
                        ds_ldmatrix(qf, qrow + ks * 64);
                        W4Num<bf16>::mma(e[0], qf[0], 0u, qf[1], 0u, kf[0], kf[1]);
                        W4Num<bf16>::mma(e[1], qf[2], 0u, qf[3], 0u, kf[2], kf[3]);
                    }
                    float sc[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int slot = tile * 8 + 2 * t + k;
                        const int pid = slot < cnt ? pages[page_of(rb + slot) - lp0] : -1;
                        sc[k] = pid >= 0 && pid < l.num_pages ? (e[0][k] + e[1][k]) * scale2 : -CUDART_INF_F;
                    }
                    float mx = fmaxf(sc[0], sc[1]);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    mx = fmaxf(mx, DS_NEG);  // a tile in which nothing is seen: probabilities 0, not NaN
                    const float p0 = ds_exp2(sc[0] - mx), p1 = ds_exp2(sc[1] - mx);
                    float ls = p0 + p1;
                    ls += __shfl_xor_sync(0xffffffffu, ls, 1);
                    ls += __shfl_xor_sync(0xffffffffu, ls, 2);
                    if (g < Gq) {
                        *reinterpret_cast<float2 *>(s_s + g * a.kv_tokens + tile * 8 + 2 * t) = make_float2(p0, p1);
                        if (t == 0) st_s[g * 32 + tile] = mx, st_s[128 + g * 32 + tile] = ls;
                    }
                }
                __syncthreads();
                if (oh < Gq) {
                    const int ntile = (cnt + 7) >> 3;
                    float m_r = lane < ntile ? st_s[oh * 32 + lane] : DS_NEG;  // lane = tile
                    m_r = warp_max(m_r);
                    const float w_tile = lane < ntile ? ds_exp2(st_s[oh * 32 + lane] - m_r) : 0.f;
                    const float l_r = warp_sum(lane < ntile ? st_s[128 + oh * 32 + lane] * w_tile : 0.f);
                    float part[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    uint32_t vrow = kv_b + sub * DS_KV_STRIDE + 256 + d8 * 16;
                    const float *prow = s_s + oh * a.kv_tokens + sub;
#pragma unroll 2
                    for (int tile = 0; tile < ntile; ++tile) {
                        const float pr = prow[tile * 8] * __shfl_sync(0xffffffffu, w_tile, tile);
                        uint4 vr = ds_lds(vrow + tile * (8 * DS_KV_STRIDE));
                        if (pr == 0.f) vr = make_uint4(0u, 0u, 0u, 0u);  // slots that are not seen hold no row
                        const float2 f0 = unpack2<bf16>(vr.x), f1 = unpack2<bf16>(vr.y), f2 = unpack2<bf16>(vr.z), f3 = unpack2<bf16>(vr.w);
                        part[0] += pr * f0.x, part[1] += pr * f0.y, part[2] += pr * f1.x, part[3] += pr * f1.y;
                        part[4] += pr * f2.x, part[5] += pr * f2.y, part[6] += pr * f3.x, part[7] += pr * f3.y;
                    }
                    // the sum over the 8 tokens of a tile position: each exchange halves the columns a lane still carries
#pragma unroll
                    for (int n = 4; n > 0; n >>= 1)
#pragma unroll
                        for (int i = 0; i < n; ++i) {
                            const bool up = sub & n;
                            const float send = up ? part[i] : part[i + n], keep = up ? part[i + n] : part[i];
                            part[i] = keep + __shfl_xor_sync(0xffffffffu, send, n);
                        }
                    const float nm = fmaxf(m_run, m_r);
                    const float fr = ds_exp2(m_run - nm), fn = ds_exp2(m_r - nm);
                    o_run = o_run * fr + part[0] * fn;
                    l_run = l_run * fr + l_r * fn;
                    m_run = nm;
                }
            }
            unsigned char *const y = x + a.o_y + (static_cast<size_t>(ab) * (q_w / 2) + kvh * Gq * 64) * 8;  // the group's heads
            if (splits == 1) {
                // o's activations go where the values lie: a warp that is done (or has no head) must not stage heads of other CTAs over rows that
                // another warp still reads.  (With more splits the merge's barrier stands between.)
                __syncthreads();
                if (oh < Gq) {
                    const float v = l_run == 0.f ? 0.f : o_run * (1.0f / l_run);
                    const float next = __shfl_down_sync(0xffffffffu, v, 1);
                    if ((sub & 1) == 0) ds_st(y + (oh * 64 + d8 * 4 + (sub >> 1)) * 8, pack2<bf16>(v, next), tag);
                }
            } else {
                unsigned char *const parts = x + a.o_part + static_cast<size_t>(item) * a.nsplit * Gq * DS_PART * 8;
                if (oh < Gq) {
                    unsigned char *const mine = parts + (split * Gq + oh) * (DS_PART * 8);
                    ds_st(mine + (d8 * 8 + sub) * 8, __float_as_uint(o_run), tag);
                    if (d8 == 0 && sub < 2) ds_st(mine + (DS_HEAD + sub) * 8, __float_as_uint(sub == 0 ? m_run : l_run), tag);
                }
                // merge: quarter heads are dealt to the splits' CTAs; a warp weighs one split's part of one quarter
                const int quarters = 4 * Gq;
                const int mine = split < quarters ? static_cast<int>((quarters - split + splits - 1) * by_splits >> 16) : 0;
#pragma unroll 1
                for (int p = warp; p < mine * splits; p += DS_WARPS) {
                    const int ui = static_cast<int>(p * by_splits >> 16), j = p - ui * splits, u = split + ui * splits, head = u >> 2;
                    const unsigned char *const po = parts + (j * Gq + head) * (DS_PART * 8) + ((u & 3) * 32 + lane) * 8;
                    const unsigned char *const pm = parts + (min(lane, splits - 1) * Gq + head) * (DS_PART * 8) + DS_HEAD * 8;
                    unsigned long long o = ds_ld(po);
                    ulonglong2 ml = ds_ld2(pm);
#pragma unroll 1
                    for (uint32_t spins = 0; ds_tag(o) != tag || ds_tag(ml.x) != tag || ds_tag(ml.y) != tag;) {
                        if (!ds_again(spins, dead)) {
                            o = ml.x = ml.y = 0x7fffffffu;
                            break;
                        }
                        o = ds_ld(po), ml = ds_ld2(pm);
                    }
                    __syncwarp();
                    const float mj = lane < splits ? __uint_as_float(static_cast<uint32_t>(ml.x)) : DS_NEG;
                    const float top = warp_max(mj);
                    const float f = lane < splits ? ds_exp2(mj - top) : 0.f;
                    const float sum = warp_sum(f * __uint_as_float(static_cast<uint32_t>(ml.y)));
                    red[p * 32 + lane] = __uint_as_float(static_cast<uint32_t>(o)) * __shfl_sync(0xffffffffu, f, j);
                    if (j == 0 && lane == 0) red_l[ui] = sum;
                }
                __syncthreads();
#pragma unroll 1
                for (int ui = warp; ui < mine; ui += DS_WARPS) {
                    float v = 0.f;
#pragma unroll 4
                    for (int j = 0; j < splits; ++j) v += red[(ui * splits + j) * 32 + lane];
                    const float sum = red_l[ui];
                    v = sum == 0.f ? 0.f : v / sum;
                    const float next = __shfl_down_sync(0xffffffffu, v, 1);
                    const int u = split + ui * splits;
                    if ((lane & 1) == 0) ds_st(y + ((u >> 2) * 64 + (u & 3) * 16 + (lane >> 1)) * 8, pack2<bf16>(v, next), tag);
                }
            }
        }
    }

    // ---- logits, and the first of the largest: a thread an output, whose piece lies in the entries of a few warps
    {
        const int P = deals[4][3], rows = deals[4][2] * 16, r0 = deals[4][1] * 16;
        for (int m = 0; m < M; ++m) {
            float bv = -INFINITY;
            int bi = INT_MAX;
            for (int r = threadIdx.x; r < rows; r += DS_THREADS) {
                const int lo = (r >> 4) * P;
                float sum = 0.f;
                for (int w = 0; w < DS_WARPS; ++w) {
                    const int4 share = shares[4][w];
                    if (share.x < lo + P && share.y > lo && share.x < share.y) sum += entries[static_cast<size_t>((r >> 4) + w) * ENTRY + (r & 15) * MP + m];
                }
                bf16 v = __float2bfloat16_rn(sum);
                if (*dead) v = __ushort_as_bfloat16(0x7fffu);
                a.logits[static_cast<size_t>(m) * a.V + r0 + r] = v;
                const float f = __bfloat162float(v);
                if (f > bv) bv = f, bi = r0 + r;  // r grows: the first maximum stays
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
            }
            if (lane == 0) best_v[m][warp] = bv, best_i[m][warp] = bi;
        }
    }
    __syncthreads();
    const uint32_t tag = tag0 + a.layers;
    if (warp < M && lane == 0) {
        float bv = best_v[warp][0];
        int bi = best_i[warp][0];
        for (int w = 1; w < DS_WARPS; ++w)
            if (best_v[warp][w] > bv || (best_v[warp][w] == bv && best_i[warp][w] < bi)) bv = best_v[warp][w], bi = best_i[warp][w];
        unsigned char *const p = a.best + (static_cast<size_t>(cta) * M + warp) * 16;
        ds_st(p, __float_as_uint(bv), tag);
        ds_st(p + 8, *dead ? ~0u : static_cast<uint32_t>(bi), tag);
    }
    if (cta == 0) {  // the step's tokens
        if (warp < M) {
            float bv = -INFINITY;
            int bi = INT_MAX;
            bool lost_one = false;
            for (int c = lane; c < ctas; c += 32) {
                const unsigned char *p = a.best + (static_cast<size_t>(c) * M + warp) * 16;
                const unsigned long long v = ds_poll(p, tag, dead), i = ds_poll(p + 8, tag, dead);
                const float ov = __uint_as_float(static_cast<uint32_t>(v));
                const int oi = static_cast<int>(static_cast<uint32_t>(i));
                lost_one |= oi < 0 || ds_tag(v) != tag || ds_tag(i) != tag;
                if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
            }
            __syncwarp();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
            }
            lost_one = __any_sync(0xffffffffu, lost_one);
            if (lane == 0) a.next_tokens[warp] = lost_one ? -1 : bi == INT_MAX ? 0 : bi;
        }
        // every CTA has read the step number by now: its packets of this step were waited for
        if (threadIdx.x == 0) *static_cast<volatile unsigned int *>(a.seq) = epoch + 1u;
        __syncthreads();
    }
    if (threadIdx.x == 0 && *dead) atomicAdd(&g_gave_up, 1u);
    tc_settle(dead);
}

// ---- weights as units: 16 rows of the MMA x 256 columns, in the order in which the lanes hold them, their scales and biases behind them.
// Rows 0-7 of unit u of piece p are rows p * step + 0..7 of `top`, columns u * 256..; rows 8-15 those of `bottom`, `shift` rows and `across` columns on:
//   16 rows: step 16, shift 8;  gate|up: step 8, top and bottom two matrices;  8 rows, both halves of the reduction: step 8, across N / 2.
__global__ void decode_step_pack_kernel(const DsMat top, const DsMat bottom, unsigned char *out, int N, int P, long long units, int step, int shift, int across) {
    const long long unit = static_cast<long long>(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (unit >= units) return;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int p = static_cast<int>(unit / P), u = static_cast<int>(unit - static_cast<long long>(p) * P);
    uint32_t *const to = reinterpret_cast<uint32_t *>(out + unit * DS_UNIT);
    for (int k = 0; k < 4; ++k) {  // (group of 128 columns, rows 0-7 or 8-15)
        const DsMat &m = k & 1 ? bottom : top;
        const size_t row = static_cast<size_t>(p) * step + g + (k & 1 ? shift : 0);
        const int word = (u * 256 + (k & 1 ? across : 0)) / 8 + (k >> 1) * 16 + t * 4;
        for (int i = 0; i < 4; ++i) to[k * 128 + lane * 4 + i] = m.w[row * (N / 8) + word + i];
    }
    const bool low = lane & 1;  // word (lane & 3) of row lane >> 2: scales of rows 0-7, of rows 8-15, biases
    const DsMat &m = low ? bottom : top;
    const size_t at = (static_cast<size_t>(p) * step + g + (low ? shift : 0)) * (N / 128) + (u * 256 + (low ? across : 0)) / 128;
    const unsigned short *const from = static_cast<const unsigned short *>(lane & 2 ? m.b : m.s) + at;
    to[512 + lane] = from[0] | static_cast<uint32_t>(from[1]) << 16;
}

// ---- host ------------------------------------------------------------------------------------------
struct Layout {
    size_t best, xchg, total;
    unsigned int o_y, o_xo, o_act, o_xd, o_part, half;
    int nsplit;
};
Layout layout(int M, int Hq, int Hkv, int D, int ff) {
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    Layout z{};
    z.nsplit = sm_count() / (M * Hkv);
    z.nsplit = z.nsplit < 1 ? 1 : z.nsplit > DS_MAX_SPLITS ? DS_MAX_SPLITS : z.nsplit;
    size_t at = up(static_cast<size_t>(M) * (Hq + 2 * Hkv) * DS_HEAD * 4);
    z.o_y = static_cast<unsigned>(at), at += up(static_cast<size_t>(M) * Hq * DS_HEAD * 4);
    z.o_xo = static_cast<unsigned>(at), at += up(static_cast<size_t>(M) * D * 4);
    z.o_act = static_cast<unsigned>(at), at += up(static_cast<size_t>(M) * ff * 4);
    z.o_xd = static_cast<unsigned>(at), at += up(static_cast<size_t>(M) * D * 4);
    z.o_part = static_cast<unsigned>(at), at += up(static_cast<size_t>(M) * Hq * z.nsplit * DS_PART * 8);
    z.half = static_cast<unsigned>(at);
    z.best = 256;
    z.xchg = z.best + up(static_cast<size_t>(sm_count()) * M * 16);
    z.total = z.xchg + 2 * at;
    return z;
}

#ifndef DS_KV_TOKENS
#define DS_KV_TOKENS 256
#endif
constexpr size_t DS_SMEM_MAX = 220 * 1024;  // beside 5 KB of static shared memory

// A warp's ring: batches, and units of a batch.
constexpr int ds_batch(int MP) { return MP <= 2 ? 2 : 1; }
constexpr int ds_batches(int MP) { return MP <= 2 ? 2 : 3; }

// Shared memory of a launch; 0: does not fit.
size_t shared_bytes(DsArgs &a, int MP) {
    const int sms = sm_count(), widest = a.ff > a.Hq * DS_HEAD ? (a.ff > a.D ? a.ff : a.D) : (a.Hq * DS_HEAD > a.D ? a.Hq * DS_HEAD : a.D);
    auto up = [](size_t v) { return (v + 127) / 128 * 128; };
    auto most = [&](int rows, int unit) { return (rows / unit + sms - 1) / sms; };
    const int unit = 8;
    int pieces = most(a.V, 16);
    pieces = pieces > most(2 * a.ff, 16) ? pieces : most(2 * a.ff, 16);
    pieces = pieces > most((a.Hq + 2 * a.Hkv) * DS_HEAD, unit) ? pieces : most((a.Hq + 2 * a.Hkv) * DS_HEAD, unit);
    const size_t entries = static_cast<size_t>(pieces + DS_WARPS) * (16 * MP + 1) * 4, merge = static_cast<size_t>(16 + DS_MAX_SPLITS) * 32 * 4;
    a.own_rows = (most(a.D, unit) + 1) * unit;
    a.act_off = static_cast<int>(up(static_cast<size_t>(DS_WARPS) * ds_batch(MP) * ds_batches(MP) * DS_UNIT));
    a.asum_bytes = static_cast<int>(up(static_cast<size_t>(widest / 128) * 8 * 4));
    a.entry_bytes = static_cast<int>(up(entries > merge ? entries : merge));
    a.kv_off = static_cast<int>(a.act_off + up(static_cast<size_t>(a.D) * (MP == 1 ? 4 : 2 * MP)));
    const size_t per = MP == 1 ? 4 : 2 * MP;  // bytes of a staged column: four columns of digits, or bf16
    const size_t wide = widest * per;
    for (a.kv_tokens = DS_KV_TOKENS; a.kv_tokens >= DS_SPLIT_TOKENS; a.kv_tokens -= 32) {
        const size_t under = a.kv_off - a.act_off + static_cast<size_t>(a.kv_tokens) * DS_KV_STRIDE;
        a.act_bytes = static_cast<int>(up(under > wide ? under : wide));
        const size_t total = a.act_off + a.act_bytes + 2u * a.asum_bytes + a.entry_bytes + 2u * a.D + static_cast<size_t>(MP) * a.own_rows * 4 + 4u * a.kv_tokens * 4 + (a.kv_tokens + 8u) * 4;
        if (total <= DS_SMEM_MAX) return total;
    }
    return 0;
}

template <int MP>
int launch(const DsArgs &a, size_t smem, cudaStream_t st) {
    static PerDevice configured;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return fail(TL_ECUDA, "decode_step: no device");
    if (!configured(device, [] { return cudaFuncSetAttribute(decode_step_kernel<MP, ds_batch(MP), ds_batches(MP)>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(DS_SMEM_MAX)) == cudaSuccess; }))
        return fail(TL_ECUDA, "decode_step: cannot raise shared memory limit");
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // the CTAs wait on one another: all are resident or the launch fails
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(sm_count());
    cfg.blockDim = dim3(DS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_step_kernel<MP, ds_batch(MP), ds_batches(MP)>, a);
    if (e != cudaSuccess) return fail(TL_ECUDA, "decode_step: launch failed: %s", cudaGetErrorString(e));
    TL_LAUNCH_CHECK("decode_step");
    return TL_OK;
}

bool sizes_fit(DsArgs &a, size_t *smem) {
    const int M = a.M, qkv_w = (a.Hq + 2 * a.Hkv) * DS_HEAD, sms = sm_count();
    if (M < 1 || M > 4 || a.layers < 1 || a.layers > DS_MAX_LAYERS || a.Hkv < 1 || a.Hq % a.Hkv != 0 || a.Hq / a.Hkv > 4 || M * a.Hkv > sms) return false;
    // whole units in both halves of a reduction, whole pieces, rows of gate|up in every CTA, all rows of a norm in one batch
    if (a.D < 512 || a.D % 512 != 0 || a.ff % 512 != 0 || (a.Hq * DS_HEAD) % 512 != 0 || a.V % 16 != 0 || a.V < 16) return false;
    if (2 * a.ff / 16 < sms || qkv_w / 16 < 1 || static_cast<long long>(a.V) / 16 * sms >= (1ll << 31)) return false;
    const int most_rows = 2 * a.ff > 2 * qkv_w ? 2 * a.ff : 2 * qkv_w;  // (gate|up goes in sixteens)
    if ((most_rows / 16 + sms - 1) / sms > DS_MAX_PIECES || (a.D / 8 + sms - 1) / sms > DS_MAX_PIECES) return false;
    const int MP = w4_pad_cols(M);
    if (M * a.D / 8 > 3 * DS_THREADS) return false;
    *smem = shared_bytes(a, MP);
    return *smem != 0;
}

}  // namespace

long long decode_step_gave_up() { return read_gave_up(); }

size_t decode_step_workspace(int batch, int layers, int num_heads, int num_kv_heads, int hidden, int intermediate, int vocab) {
    DsArgs a{};
    a.M = batch, a.layers = layers, a.Hq = num_heads, a.Hkv = num_kv_heads, a.D = hidden, a.ff = intermediate, a.V = vocab;
    size_t smem = 0;
    if (batch < 1 || num_heads < 1 || num_kv_heads < 1 || !sizes_fit(a, &smem)) return 0;
    return layout(batch, num_heads, num_kv_heads, hidden, intermediate).total;
}

int launch_decode_step_pack(const tl_packed_matrix &top, const tl_packed_matrix *bottom, void *out, int rows, int N, int halves, cudaStream_t st) {
    const int step = halves || bottom ? 8 : 16, P = N / (halves ? 512 : 256);
    if (rows < 1 || N < 1 || rows % step != 0 || N % (halves ? 512 : 256) != 0 || (halves && bottom) || !aligned16(out))
        return fail(TL_EINVAL, "decode_step_pack: rows in whole pieces, columns in whole units, a 16-byte aligned result");
    auto mat = [](const tl_packed_matrix &m) { return DsMat{static_cast<const uint32_t *>(m.weight), m.scales, m.biases}; };
    const long long units = static_cast<long long>(rows / step) * P;
    decode_step_pack_kernel<<<static_cast<unsigned>((units + 7) / 8), 256, 0, st>>>(mat(top), mat(bottom ? *bottom : top), static_cast<unsigned char *>(out), N, P, units, step,
                                                                                     halves || bottom ? 0 : 8, halves ? N / 2 : 0);
    TL_LAUNCH_CHECK("decode_step_pack");
    return TL_OK;
}

int launch_decode_step(const tl_decode_step_plan &p, cudaStream_t st) {
    static_assert(sizeof(DsArgs) < 32 * 1024, "kernel parameters");
    DsArgs a{};
    a.M = p.batch, a.layers = p.layers, a.Hq = p.num_heads, a.Hkv = p.num_kv_heads, a.D = p.hidden, a.ff = p.intermediate, a.V = p.vocab;
    size_t smem = 0;
    if (!sizes_fit(a, &smem)) return fail(TL_EINVAL, "decode_step: sizes the one-launch step does not take (tl_decode_step_workspace says 0)");
    if (static_cast<unsigned long long>(p.page_size) * p.page_size * p.max_pages >= (1ull << 32))
        return fail(TL_EINVAL, "decode_step: max_pages x page_size x page_size must stay below 2^32");
    const Layout z = layout(a.M, a.Hq, a.Hkv, a.D, a.ff);
    if (p.workspace_bytes < z.total) return fail(TL_EWORKSPACE, "decode_step: workspace too small");
    a.nsplit = z.nsplit;
    a.page_size = p.page_size, a.page_inverse = static_cast<unsigned>((0xffffffffull + p.page_size) / p.page_size), a.max_pages = p.max_pages, a.norm_eps = p.norm_eps;
    a.tokens = p.tokens, a.offsets = p.offsets, a.context_lens = p.context_lens, a.inv_freq = p.rope_inv_freq;
    a.emb = DsMat{static_cast<const uint32_t *>(p.embedding.weight), p.embedding.scales, p.embedding.biases};
    a.head = static_cast<const unsigned char *>(p.head), a.norm = static_cast<const bf16 *>(p.norm);
    a.logits = static_cast<bf16 *>(p.logits), a.next_tokens = p.next_tokens;
    unsigned char *ws = static_cast<unsigned char *>(p.workspace);
    a.seq = reinterpret_cast<unsigned int *>(ws);
    a.best = ws + z.best;
    a.xchg[0] = ws + z.xchg, a.xchg[1] = ws + z.xchg + z.half;
    a.o_y = z.o_y, a.o_xo = z.o_xo, a.o_act = z.o_act, a.o_xd = z.o_xd, a.o_part = z.o_part;
    bool ok = aligned16(ws) && aligned16(a.head) && aligned16(a.norm);
    for (int i = 0; i < a.layers; ++i) {
        const tl_decode_step_layer &from = p.layer[i];
        DsLayer &to = a.layer[i];
        const void *const w[4] = {from.qkv, from.o, from.gate_up, from.down};
        for (int k = 0; k < 4; ++k) to.w[k] = static_cast<const unsigned char *>(w[k]), ok = ok && aligned16(w[k]);
        to.ln1 = static_cast<const bf16 *>(from.input_norm), to.ln2 = static_cast<const bf16 *>(from.post_norm);
        to.q_norm = static_cast<const bf16 *>(from.q_norm), to.k_norm = static_cast<const bf16 *>(from.k_norm);
        to.k_pages = static_cast<bf16 *>(from.key_pages), to.v_pages = static_cast<bf16 *>(from.value_pages), to.table = from.block_table;
        to.num_pages = from.num_pages;
        to.ln1_eps = from.input_eps, to.ln2_eps = from.post_eps, to.q_eps = from.q_eps, to.k_eps = from.k_eps, to.scale = from.scale;
        ok = ok && aligned16(to.ln1) && aligned16(to.ln2) && aligned16(to.k_pages) && aligned16(to.v_pages) &&
             ((reinterpret_cast<uintptr_t>(to.q_norm) | reinterpret_cast<uintptr_t>(to.k_norm)) & 3u) == 0;
    }
    if (!ok) return fail(TL_EINVAL, "decode_step: operands must be 16-byte aligned");
    switch (w4_pad_cols(a.M)) {
        case 1: return launch<1>(a, smem, st);
        case 2: return launch<2>(a, smem, st);
        default: return launch<4>(a, smem, st);
    }
}

}  // namespace tl
