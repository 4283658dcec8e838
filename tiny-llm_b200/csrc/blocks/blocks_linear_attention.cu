// Linear attention with a decay (a recurrent mixer) over ragged batches, its state kept in fp32 slots.
//
// Per sequence and head a matrix S [dk, dv] is carried from token to token:
//     S <- diag(alpha_t) S + k_t v_t^T,      o_t = S^T (q_scale * q_t),
//     alpha_t = sigmoid(z_t + bias)^(1 / tau) = exp(log_sigmoid(z_t + bias) / tau)        (per key channel)
// or, given head_decay, one fixed alpha per head (retention).  With rotation tables the first rope_dims entries of every
// head of q and k are rotated by the token's tabulated angle while they are staged, in fp32: what enters the recurrence is
// never rounded back to the projections' type.
// The columns of S never mix, so a CTA owns 32 (64, 128) of them for one (sequence, head) and walks tokens in order; 4 lanes share
// one (two, four) columns, each holding every 4th row of them in registers.  The tokens' q, k and decays are staged 16 (8 for dk > 128) at a time in shared
// memory as fp32 (the decay is computed there, in fp32, from the fp32 logits).  A sequence that starts at position 0
// starts from zero, whatever its slot held; otherwise the slot is read, and in both cases written back after the last
// token.  Single tokens and portions of up to 64 tokens are one walk.  A longer portion is cut into segments at the
// multiples of 64 in ABSOLUTE positions, which run side by side in three launches: every segment's outputs and end state from a
// zero state (the first one from the sequence's own), with its queries times the decays since its start put aside; the start state
// of every segment by walking those in order (S' = decay * S + local); and what a start state adds to its segment's outputs, the
// product of those queries with it.  (The recurrence run once more from the start states instead of that product was half of
// the time.)  Every sum has an order fixed by token, channel and segment
// indices alone; the cuts depend on positions only, so how a prompt was cut into steps changes the result by the
// rounding of the combination at most.
// 2048 tokens in two sequences, 16 heads of 64 x 128: 208 + 9 + 208 us (the recurrence twice, a column a thread) -> 99 + 19 + 24.
// The scan is bound by instructions and the staging's round trips: 25 M of its 50 M are multiply-adds.  Long portions with a decay per key channel take
// the tensor cores instead (decay_chunk_kernel below).
#include <type_traits>

#include "blocks_common.cuh"

namespace tlb {

constexpr int kLaThreads = 128;
constexpr int kLaLanes = 4;    // lanes per column
constexpr int kLaSegment = TLB_DECAY_SCAN_SEGMENT;  // positions per segment of a long portion

// Segment c of a sequence's new tokens [p0, p0 + n): cut at the multiples of kLaSegment in ABSOLUTE positions, so that
// where a prompt was cut into steps does not move the cuts.  Returns false when the sequence has no segment c.
__device__ __forceinline__ bool la_segment(int p0, int n, int c, int &lo, int &hi, int &nseg) {
    const int end = p0 + n, b0 = (p0 / kLaSegment + 1) * kLaSegment;
    nseg = (n <= kLaSegment || end <= b0) ? 1 : 1 + (end - b0 + kLaSegment - 1) / kLaSegment;  // a short portion is never cut
    if (c >= nseg) return false;
    lo = c == 0 ? p0 : b0 + (c - 1) * kLaSegment;
    hi = nseg == 1 ? end : min(end, c == 0 ? b0 : lo + kLaSegment);
    return true;
}

// One kernel, two uses (SEG):
//   0  the whole portion of a sequence in one CTA per (head, column block): state from the slot (or zero at position 0),
//      outputs, state back to the slot.  Single tokens and short portions.
//   1  segment c alone, from a ZERO state (c = 0: as in the first use): its outputs, and to the workspace its end state, the product of
//      its decays and (c > 0) its scaled queries times the decays from its first token on, decayed [T, heads, dk]; of a
//      sequence's last segment also the steps themselves, last_steps [sequences, 64, heads, dk] = (decay, key).  A sequence that
//      is one segment is done with that.
//
// decay_kind chooses where the decay comes from: 0 = sigmoid(z + bias)^(1/tau) per key channel, or head_decay; 2 = exp(-exp(z + bias))
// per key channel; 3 = one number per head and token, exp(-exp(a_log[h]) dt) with dt = softplus(z[t, h] + bias[h]), and the
// token's key is multiplied by dt (a discretised state-space step); 4 = one (decay, key factor) pair per head and token as given
// by z [T, heads, 2] (a gated memory whose log weights were stabilised beforehand).  Columns of the state from v_cols up have
// no value: v is 1 there, so that column v_cols carries the decayed sum of the keys themselves (a normaliser).  q and k may have fewer heads than v (qk_heads; head h
// reads query/key head h / (heads / qk_heads)).  skip [heads]: o_t += skip[h] v_t.  BONUS: the read-out comes BEFORE the
// update and sees the token's own k v^T weighted by bonus [heads, dk] instead: o_t = (S + diag(bonus) k_t v_t^T)^T q_t.
// SCALAR: the decay is one number per head and token (head_decay, decay_kind 3 and 4): it is read once per token, and a row of the
// state reads 8 bytes of its token's staged numbers instead of 16.
// NC: state columns per thread.  A row's staged numbers are read from shared memory once for all of them: with one column the scan
// was bound by those reads (16 bytes for three multiply-adds, and every 32 columns staged the decays anew).
// One column a thread is the form of decoding steps, a wave of CTAs that load their state, take a token and store it, and of short
// portions: as many CTAs to an SM as fitted before it had staging in batches (16 rows a lane: 160 registers without a bound, three
// CTAs; 16 tokens of 8 heads of 64 x 128 then took two waves: 5.5 us became 7.4, with the bound 5.1).  With one decay per head and 32
// rows a lane eight CTAs an SM leave 64 registers, which staging in batches spilled: up to three times the time of the plain walk.
// So there the entries are staged one at a time, and it is seven (six for segments).  8 heads of 128 x 256, one decay per head: 64 tokens of
// one sequence 48 us as a plain walk, 152 spilled, 39 now; 16 sequences of a token 9.6, 11.6, 8.4.
template <typename T, int KR /* rows per lane: dk <= 4 * KR */, int kLaTokens /* tokens staged at a time */, bool BONUS, bool SCALAR, int NC, bool SEG>
__global__ void __launch_bounds__(kLaThreads, NC > 1 ? (KR == 32 ? 3 : 4) : SCALAR && KR == 32 ? (SEG ? 6 : 7) : KR == 8 ? 5 : KR == 16 ? 4 : 1)
decay_scan_kernel(const T *__restrict__ q, long long q_token, long long q_head, const T *__restrict__ k, long long k_token, long long k_head,
                  const T *__restrict__ v, long long v_token, long long v_head, const float *__restrict__ z, long long z_token,
                  const T *__restrict__ z_bias, float inv_tau, const float *__restrict__ head_decay, const float *__restrict__ rope_cos,
                  const float *__restrict__ rope_sin, int rope_dims, int rope_interleaved, float q_scale, int heads, int dk, int dv,
                  const int32_t *__restrict__ seq_info,
                  float *__restrict__ state, long long slot_stride, int num_slots, float *__restrict__ out, int max_segments,
                  float *__restrict__ seg_state, float *__restrict__ seg_decay, float *__restrict__ decayed, float2 *__restrict__ last_steps, int decay_kind, const T *__restrict__ a_log,
                  const T *__restrict__ bonus, int qk_heads, const T *__restrict__ skip, int v_cols) {
    __shared__ float4 sx[SCALAR ? 1 : kLaTokens * 4 * KR];   // per token and key channel: (decay, k, scaled q, k times the bonus), one 16-byte read per row
    __shared__ float2 skq[SCALAR ? kLaTokens * 4 * KR : 1];  // SCALAR: (k, scaled q)
    constexpr int COLS = kLaThreads / kLaLanes * NC;  // per CTA
    constexpr int BATCH = NC == 1 && SCALAR && KR == 32 ? 1 : 4, VALUES = BATCH == 1 ? 1 : 8;
    __shared__ __align__(16) float sv[kLaTokens * COLS];
    __shared__ float sprod[4 * KR];
    __shared__ float2 s_step[kLaTokens];  // SCALAR: the token's (decay, key factor), worked out or read once per token
    __shared__ float2 s_chan[4 * KR];     // per key channel of this head: (the decay logit's bias, the bonus), read once
    const int colblocks = (dv + COLS - 1) / COLS;
    const int s = blockIdx.x, head = blockIdx.y / colblocks, col0 = (blockIdx.y % colblocks) * COLS, c = blockIdx.z;
    const int seq_first = seq_info[s * 4 + 0], seq_count = seq_info[s * 4 + 1], start = seq_info[s * 4 + 2], slot = seq_info[s * 4 + 3];
    int lo = start, hi = start + seq_count, nseg = 1;
    if (SEG && !la_segment(start, seq_count, c, lo, hi, nseg)) return;
    const int first = seq_first + (lo - start), count = hi - lo;
    const int cidx = threadIdx.x / kLaLanes, r = threadIdx.x % kLaLanes;
    const int col = col0 + cidx * NC;  // .. col + NC - 1
    const int cols = min(NC, dv - col);  // <= 0: none
    const bool slot_ok = slot >= 0 && slot < num_slots;
    float *mine = state + (size_t)(slot_ok ? slot : 0) * slot_stride + (size_t)head * dk * dv;
    float *seg = SEG ? seg_state + (((size_t)s * max_segments + c) * heads + head) * dk * dv : nullptr;
    const bool from_slot = !SEG || c == 0;  // else from zero
    const bool to_slot = !SEG || nseg == 1;
    const bool keeps_decays = SEG && !to_slot && col0 == 0;  // one column block per head

    const bool has_state = from_slot && lo > 0 && slot_ok;
    float S[KR][NC];
#pragma unroll
    for (int i = 0; i < KR; ++i) {
        const int row = r + kLaLanes * i;
#pragma unroll
        for (int u = 0; u < NC; ++u) S[i][u] = has_state && row < dk && u < cols ? mine[(size_t)row * dv + col + u] : 0.f;
    }
    if (keeps_decays)
        for (int d = threadIdx.x; d < dk; d += blockDim.x) sprod[d] = 1.f;
    for (int d = threadIdx.x; d < dk; d += blockDim.x)
        s_chan[d] = make_float2((z_bias && decay_kind < 3) ? to_f(z_bias[(size_t)head * dk + d]) : 0.f, BONUS ? to_f(bonus[(size_t)head * dk + d]) : 0.f);
    const int qk_head = head / (heads / qk_heads);
    const float rate = decay_kind == 3 ? expf(to_f(a_log[head])) : 0.f;
    const float skipv = skip ? to_f(skip[head]) : 0.f;
    for (int t0 = 0; t0 < count; t0 += kLaTokens) {
        const int n = min(kLaTokens, count - t0);
        __syncthreads();
        if (SCALAR && decay_kind == 3) {
            if (threadIdx.x < n) {
                const float zz = z[(size_t)(first + t0 + threadIdx.x) * z_token + head] + (z_bias ? to_f(z_bias[head]) : 0.f);
                const float dt = zz > 20.f ? zz : log1pf(expf(zz));
                s_step[threadIdx.x] = make_float2(expf(-rate * dt), dt);
            }
            __syncthreads();
        } else if (SCALAR) {
            if (threadIdx.x < n)
                s_step[threadIdx.x] = decay_kind == 4 ? *reinterpret_cast<const float2 *>(z + (size_t)(first + t0 + threadIdx.x) * z_token + 2 * head)
                                                      : make_float2(head_decay[head], 1.f);
            __syncthreads();
        }
        // BATCH entries' numbers are on their way at once: one at a time, a chunk's staging was a chain of memory round trips longer
        // than its multiply-adds
        for (int e0 = threadIdx.x; e0 < n * dk; e0 += BATCH * kLaThreads) {
            float zs[BATCH];
            T ks[BATCH], qs[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int e = e0 + u * kLaThreads;
                if (e >= n * dk) break;
                const int j = e / dk, d = e - j * dk;
                const size_t tok = (size_t)(first + t0 + j);
                if (!SCALAR) zs[u] = z[tok * z_token + (size_t)head * dk + d];
                ks[u] = k[tok * k_token + (size_t)qk_head * k_head + d], qs[u] = q[tok * q_token + (size_t)qk_head * q_head + d];
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int e = e0 + u * kLaThreads;
                if (e >= n * dk) break;
                const int j = e / dk, d = e - j * dk;
                const size_t tok = (size_t)(first + t0 + j);
                float alpha, kmul = 1.f;
                if (SCALAR) alpha = 0.f, kmul = s_step[j].y;
                else if (decay_kind == 2) alpha = expf(-expf(zs[u] + s_chan[d].x));
                else alpha = expf(log_sigmoid(zs[u] + s_chan[d].x) * inv_tau);
                float kd = to_f(ks[u]), qd = to_f(qs[u]);
                if (d < rope_dims) {  // rotate the pair this entry belongs to, in fp32, by the token's tabulated angle
                    const int half = rope_dims >> 1;
                    const bool low = rope_interleaved ? !(d & 1) : d < half;
                    const int i = rope_interleaved ? d >> 1 : (low ? d : d - half);
                    const int other = rope_interleaved ? (d ^ 1) : (low ? d + half : d - half);
                    const float c = rope_cos[tok * half + i], sn = low ? -rope_sin[tok * half + i] : rope_sin[tok * half + i];
                    kd = kd * c + to_f(k[tok * k_token + (size_t)qk_head * k_head + other]) * sn;
                    qd = qd * c + to_f(q[tok * q_token + (size_t)qk_head * q_head + other]) * sn;
                }
                kd *= kmul;
                if (SCALAR) skq[j * 4 * KR + d] = make_float2(kd, qd * q_scale);
                else sx[j * 4 * KR + d] = make_float4(alpha, kd, qd * q_scale, BONUS ? kd * s_chan[d].y : 0.f);
            }
        }
        for (int e0 = threadIdx.x; e0 < n * COLS; e0 += VALUES * kLaThreads) {
            T vs[VALUES];
#pragma unroll
            for (int u = 0; u < VALUES; ++u) {
                const int e = e0 + u * kLaThreads, j = e / COLS, d = e - j * COLS;
                if (e < n * COLS && col0 + d < v_cols) vs[u] = v[(size_t)(first + t0 + j) * v_token + (size_t)head * v_head + col0 + d];
            }
#pragma unroll
            for (int u = 0; u < VALUES; ++u) {
                const int e = e0 + u * kLaThreads, d = e % COLS;
                if (e < n * COLS) sv[e] = col0 + d < v_cols ? to_f(vs[u]) : col0 + d < dv ? 1.f : 0.f;
            }
        }
        __syncthreads();
        if (keeps_decays) {  // the segment's decay product per key channel, in token order, and the queries times it
            for (int d = threadIdx.x; d < dk; d += blockDim.x) {
                float p = sprod[d];
                for (int j = 0; j < n; ++j) {
                    const float before = p;
                    p *= SCALAR ? s_step[j].x : sx[j * 4 * KR + d].x;
                    if (c == nseg - 1)
                        last_steps[(((size_t)s * kLaSegment + t0 + j) * heads + head) * dk + d] =
                            SCALAR ? make_float2(s_step[j].x, skq[j * 4 * KR + d].x) : make_float2(sx[j * 4 * KR + d].x, sx[j * 4 * KR + d].y);
                    if (c > 0)
                        decayed[((size_t)(first + t0 + j) * heads + head) * dk + d] = (SCALAR ? skq[j * 4 * KR + d].y : sx[j * 4 * KR + d].z) * (BONUS ? before : p);
                }
                sprod[d] = p;
            }
        }
        for (int j = 0; j < n; ++j) {
            float vj[NC];
            if constexpr (NC >= 4) {
#pragma unroll
                for (int u = 0; u < NC; u += 4) *reinterpret_cast<float4 *>(vj + u) = *reinterpret_cast<const float4 *>(sv + j * COLS + cidx * NC + u);
            } else if constexpr (NC == 2) *reinterpret_cast<float2 *>(vj) = *reinterpret_cast<const float2 *>(sv + j * COLS + cidx * NC);
            else vj[0] = sv[j * COLS + cidx];
            const float4 *xa = sx + (SCALAR ? 0 : j * 4 * KR);
            const float2 *ya = skq + (SCALAR ? j * 4 * KR : 0);
            const float keep = SCALAR ? s_step[j].x : 0.f;
            auto staged = [&](int row) {
                if (!SCALAR) return xa[row];
                const float2 y = ya[row];
                return make_float4(keep, y.x, y.y, 0.f);
            };
            float o[2][NC] = {};  // over this lane's even and odd rows
            auto rows = [&](auto whole) {  // whole: dk = 4 KR, no row to leave out
#pragma unroll
                for (int i = 0; i < KR; ++i) {
                    const int row = r + kLaLanes * i;
                    if (decltype(whole)::value || row < dk) {
                        const float4 x = staged(row);
#pragma unroll
                        for (int u = 0; u < NC; ++u) {
                            if (BONUS) o[i & 1][u] = fmaf(x.z, fmaf(x.w, vj[u], S[i][u]), o[i & 1][u]);
                            S[i][u] = fmaf(x.x, S[i][u], x.y * vj[u]);
                            if (!BONUS) o[i & 1][u] = fmaf(x.z, S[i][u], o[i & 1][u]);
                        }
                    }
                }
            };
            if ((NC > 1 || KR <= 16 || SCALAR) && dk == 4 * KR) rows(std::true_type{});
            else rows(std::false_type{});
            // the four lanes' sums: ((0 + 1) + (2 + 3)), each lane ending with its share of the columns
            float *to = out + ((size_t)(first + t0 + j) * heads + head) * dv + col;
            if constexpr (NC == 4) {
                const bool odd = r & 1, high = r & 2;
                float y[4], w[2];
#pragma unroll
                for (int u = 0; u < 4; ++u) y[u] = o[0][u] + o[1][u];
#pragma unroll
                for (int u = 0; u < 2; ++u) {  // columns u and u + 2 of this lane's parity: 0, 2 or 1, 3
                    const float keep_y = odd ? y[2 * u + 1] : y[2 * u], give = odd ? y[2 * u] : y[2 * u + 1];
                    w[u] = keep_y + __shfl_xor_sync(0xffffffffu, give, 1);
                }
                const float mine_y = high ? w[1] : w[0], give = high ? w[0] : w[1];
                const float sum = mine_y + __shfl_xor_sync(0xffffffffu, give, 2);
                const float vr = r == 0 ? vj[0] : r == 1 ? vj[1] : r == 2 ? vj[2] : vj[3];
                if (r < cols) to[r] = fmaf(skipv, vr, sum);
            } else {
#pragma unroll
                for (int u = 0; u < NC; ++u) {
                    float y = o[0][u] + o[1][u];
                    y += __shfl_xor_sync(0xffffffffu, y, 1);
                    y += __shfl_xor_sync(0xffffffffu, y, 2);
                    if (u < cols && r == u) to[u] = fmaf(skipv, vj[u], y);
                }
            }
        }
    }
    float *dst = to_slot ? (slot_ok ? mine : nullptr) : seg;
    if (dst != nullptr) {
#pragma unroll
        for (int i = 0; i < KR; ++i) {
            const int row = r + kLaLanes * i;
#pragma unroll
            for (int u = 0; u < NC; ++u)
                if (row < dk && u < cols) dst[(size_t)row * dv + col + u] = S[i][u];
        }
    }
    if (keeps_decays) {
        __syncthreads();
        float *pd = seg_decay + (((size_t)s * max_segments + c) * heads + head) * dk;
        for (int d = threadIdx.x; d < dk; d += blockDim.x) pd[d] = sprod[d];
    }
}

// Walk a sequence's segments in order, S_start[c + 1] = decay[c] * S_start[c] + local[c], and leave every segment's START state
// where its local end state was (segment 0 began from the sequence's own state: nothing is added to it); then the last segment's
// tokens from its start state, step by step as the scan itself takes them, to the state the slot gets.  One thread per W
// neighbouring state elements of a row (W = 4: a row's numbers and the addresses are had once for four), (sequence, head) per blockIdx.
template <typename T, int W>
__global__ void __launch_bounds__(256)
decay_combine_kernel(const int32_t *__restrict__ seq_info, float *__restrict__ state, long long slot_stride, int num_slots, int heads, int dk,
                     int dv, int max_segments, float *__restrict__ seg_state, const float *__restrict__ seg_decay, const float2 *__restrict__ last_steps,
                     const T *__restrict__ v, long long v_token, long long v_head, int v_cols) {
    const int s = blockIdx.x, head = blockIdx.y;
    const int seq_first = seq_info[s * 4 + 0], count = seq_info[s * 4 + 1], start = seq_info[s * 4 + 2], slot = seq_info[s * 4 + 3];
    int lo, hi, nseg;
    la_segment(start, count, 0, lo, hi, nseg);
    if (nseg <= 1) return;
    la_segment(start, count, nseg - 1, lo, hi, nseg);
    const int n = hi - lo;
    const T *values = v + (size_t)(seq_first + lo - start) * v_token + (size_t)head * v_head;
    const float2 *steps = last_steps + ((size_t)s * kLaSegment * heads + head) * dk;
    for (int e = (blockIdx.z * blockDim.x + threadIdx.x) * W; e < dk * dv; e += gridDim.z * blockDim.x * W) {
        const int row = e / dv, col = e - row * dv;
        float S[W] = {};
        // eight segments' local states and decays (tokens' steps) are fetched before the first of them is used: the walk is a
        // chain of multiply-adds, not of memory round trips
        constexpr int kAhead = 8;
        float *seg = seg_state + ((size_t)s * max_segments * heads + head) * dk * dv + e;
        const float *dec = seg_decay + ((size_t)s * max_segments * heads + head) * dk + row;
        const size_t seg_step = (size_t)heads * dk * dv, dec_step = (size_t)heads * dk;
        for (int c0 = 0; c0 < nseg; c0 += kAhead, seg += kAhead * seg_step, dec += kAhead * dec_step) {
            float local[kAhead][W], decay[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (c0 + u + 1 < nseg) {
                    if constexpr (W == 4) *reinterpret_cast<float4 *>(local[u]) = *reinterpret_cast<const float4 *>(seg + u * seg_step);
                    else local[u][0] = seg[u * seg_step];
                    decay[u] = dec[u * dec_step];
                }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (c0 + u < nseg) {
                    if constexpr (W == 4) *reinterpret_cast<float4 *>(seg + u * seg_step) = make_float4(S[0], S[1], S[2], S[3]);
                    else seg[u * seg_step] = S[0];
                    if (c0 + u + 1 < nseg) {
#pragma unroll
                        for (int w = 0; w < W; ++w) S[w] = fmaf(decay[u], S[w], local[u][w]);
                    }
                }
        }
        if (slot < 0 || slot >= num_slots) continue;
        const float2 *step = steps + row;
        const T *value = values + col;
        for (int t0 = 0; t0 < n; t0 += kAhead, step += kAhead * dec_step, value += kAhead * v_token) {
            float2 x[kAhead];
            T vj[kAhead][W];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (t0 + u < n) {
                    x[u] = step[u * dec_step];
#pragma unroll
                    for (int w = 0; w < W; ++w)
                        if (col + w < v_cols) vj[u][w] = value[u * v_token + w];
                }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (t0 + u < n) {
#pragma unroll
                    for (int w = 0; w < W; ++w) S[w] = fmaf(x[u].x, S[w], x[u].y * (col + w < v_cols ? to_f(vj[u][w]) : 1.f));
                }
        }
        float *to = state + (size_t)slot * slot_stride + (size_t)head * dk * dv + e;
#pragma unroll
        for (int w = 0; w < W; ++w) to[w] = S[w];
    }
}

// out[t, h, :] += decayed[t, h, :] S_start for the tokens of segments 1, 2, ..: a product of up to 64 tokens x dk by dk x 128 columns
// per CTA, in fp32, k ascending.  Thread: 8 tokens x 8 columns (two runs of four).  VEC: rows are whole 16-byte pieces.
constexpr int kLaOutCols = 128, kLaOutK = 32;
template <bool VEC>
__global__ void __launch_bounds__(128)
decay_output_kernel(const int32_t *__restrict__ seq_info, int heads, int dk, int dv, int max_segments, const float *__restrict__ seg_state,
                    const float *__restrict__ decayed, float *__restrict__ out) {
    const int colblocks = (dv + kLaOutCols - 1) / kLaOutCols;
    const int s = blockIdx.x, head = blockIdx.y / colblocks, col0 = (blockIdx.y % colblocks) * kLaOutCols, c = blockIdx.z + 1;
    const int seq_first = seq_info[s * 4 + 0], count = seq_info[s * 4 + 1], start = seq_info[s * 4 + 2];
    int lo, hi, nseg;
    if (!la_segment(start, count, c, lo, hi, nseg)) return;
    const int first = seq_first + (lo - start), n = hi - lo;
    const float *S = seg_state + (((size_t)s * max_segments + c) * heads + head) * dk * dv + col0;
    const float *Q = decayed + ((size_t)first * heads + head) * dk;
    __shared__ __align__(16) float sq[kLaOutK][kLaSegment + 4], ss[kLaOutK][kLaOutCols];
    const int tr = threadIdx.x / 16 * 8, tc = threadIdx.x % 16 * 4;
    float acc[8][8] = {};
    for (int k0 = 0; k0 < dk; k0 += kLaOutK) {
        float4 q4[4], s4[8];
        auto piece = [&](const float *p, int left) {  // up to four entries of a row, zeros past its end
            if (VEC) return left > 0 ? *reinterpret_cast<const float4 *>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
            return make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
        };
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // 64 tokens x 8 pieces of k
            const int e = threadIdx.x + i * 128, t = e / 8, k = k0 + e % 8 * 4;
            q4[i] = piece(Q + (size_t)t * heads * dk + k, t < n ? dk - k : 0);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {  // 32 k x 32 pieces of columns
            const int e = threadIdx.x + i * 128, k = k0 + e / 32, d = e % 32 * 4;
            s4[i] = piece(S + (size_t)k * dv + d, k < dk ? dv - col0 - d : 0);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 128, t = e / 8, k = e % 8 * 4;
            sq[k][t] = q4[i].x, sq[k + 1][t] = q4[i].y, sq[k + 2][t] = q4[i].z, sq[k + 3][t] = q4[i].w;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = threadIdx.x + i * 128;
            *reinterpret_cast<float4 *>(&ss[e / 32][e % 32 * 4]) = s4[i];
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < kLaOutK; ++k) {
            float q[8], x[8];
            *reinterpret_cast<float4 *>(q) = *reinterpret_cast<const float4 *>(&sq[k][tr]);
            *reinterpret_cast<float4 *>(q + 4) = *reinterpret_cast<const float4 *>(&sq[k][tr + 4]);
            *reinterpret_cast<float4 *>(x) = *reinterpret_cast<const float4 *>(&ss[k][tc]);
            *reinterpret_cast<float4 *>(x + 4) = *reinterpret_cast<const float4 *>(&ss[k][tc + 64]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(q[i], x[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (tr + i >= n) break;
        float *o = out + ((size_t)(first + tr + i) * heads + head) * dv + col0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int d = tc + 64 * h;
            if (VEC) {
                if (col0 + d >= dv) continue;
                float4 y = *reinterpret_cast<const float4 *>(o + d);
                y.x += acc[i][4 * h], y.y += acc[i][4 * h + 1], y.z += acc[i][4 * h + 2], y.w += acc[i][4 * h + 3];
                *reinterpret_cast<float4 *>(o + d) = y;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (col0 + d + j < dv) o[d + j] += acc[i][4 * h + j];
            }
        }
    }
}

// ---- portions of more than a segment with a decay per key channel, on the tensor cores ------------------------------------------------
// Sixteen tokens at a time, A_t the product of the decays up to token t of the sixteen and R_s that of the decays behind token s:
//     o_t = sum_d q_t[d] A_t[d] S[d, :]  +  sum_{s <= t} P[t, s] v_s        P[t, s] = sum_d q_t[d] k_s[d] decay(s+1 .. t)[d]
//     S  <- diag(A_16) S + sum_s (k_s R_s) v_s^T
// All factors are products of decays, at most 1, whatever the decays are.  P is formed in fp32 as it stands (each token's key times the decays
// one after another); the three products run on mma.sync with fp32 sums.  Its operands are 16-bit: v is bf16 as it is; q A, k R, P and S, which are fp32, enter
// as three bf16 terms each (24 bits; of nine products of two such operands the three below 2^-24 are left out).  The tensor cores cut their sums off where a
// multiply-add rounds, so no long sum is left to them: products of 16 start from zero and are added in fp32.
// S^T [columns, channels] stays in accumulator fragments, which are the A operand's layout too: a warp owns 32 columns.
//
// Three launches: every segment's end state from zero (its first one's from the sequence's own state) and its decay (MODE 0); the segments' start states, in
// order, the first one's too; the outputs from the start states, and the last segment's end state to the slot (MODE 1).  The CTAs of a launch have no order, so
// the launch that writes the slot of a sequence in several segments does not read it.
// 2048 tokens in two sequences of 16 heads of 64 x 128: the walk in segments 99 + 19 + 24 us, this 18 + 8 + 48 (8 + 8 heads 1.6 x, 65 tokens 1.1 x, 8000
// tokens 2 x as fast); the error against 64 bits is 0.85 to 1.0 of the walk's (with long sums left to the tensor cores it was twice that, at 42 us).
// What bounds it: instructions and their latencies, with 14 warps an SM: issue slots 49 % busy (MODE 1: 2900 instructions a warp and sixteen tokens, an eighth of them for the
// terms of S), 1.8 of the 7.0 cycles between two instructions of a warp for the one before, 2.0 for loads, 0.4 at the three barriers.
constexpr int kCkTokens = 16, kCkCols = 128;

__device__ __forceinline__ void ck_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ck_ldm(uint32_t (&r)[4], const bf16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p)))
                 : "memory");
}
__device__ __forceinline__ void ck_ldm_t(uint32_t (&r)[4], const bf16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p)))
                 : "memory");
}
// x, y as three pairs of bf16: x = x0 + x1 + x2 up to 2^-24 of it
__device__ __forceinline__ void ck_split(float x, float y, uint32_t (&term)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        term[i] = tl::pack2<bf16>(x, y);
        if (i < 2) {
            const float2 f = tl::unpack2<bf16>(term[i]);
            x -= f.x, y -= f.y;
        }
    }
}

template <int DK, int MODE>
__global__ void __launch_bounds__(128, 4)
decay_chunk_kernel(const bf16 *__restrict__ q, long long q_token, long long q_head, const bf16 *__restrict__ k, long long k_token, long long k_head,
                   const bf16 *__restrict__ v, long long v_token, long long v_head, const float *__restrict__ z, long long z_token,
                   const bf16 *__restrict__ z_bias, float inv_tau, float q_scale, int heads, int dv, const int32_t *__restrict__ seq_info,
                   float *__restrict__ state, long long slot_stride, int num_slots, float *__restrict__ out, int max_segments,
                   float *__restrict__ seg_state, float *__restrict__ seg_decay, int decay_kind) {
    constexpr int ROW = DK + 8, VROW = kCkCols + 8, PROW = kCkTokens + 8, PER = DK / 8;  // padded rows (banks); channels a thread stages
    constexpr int RAW_Q = 0, RAW_K = kCkTokens * DK * 2, RAW_Z = 2 * RAW_K, RAW = RAW_Z + kCkTokens * DK * 4;
    constexpr int NT = DK / 8, KT = DK / 16;
    __shared__ __align__(16) float s_alpha[kCkTokens][DK], s_q[MODE ? kCkTokens : 1][DK], s_k[kCkTokens][DK];
    __shared__ __align__(16) bf16 t_q[MODE ? 3 : 1][kCkTokens][ROW], t_k[3][kCkTokens][ROW], t_p[MODE ? 3 : 1][kCkTokens][PROW], s_v[2][kCkTokens][VROW];
    __shared__ __align__(16) unsigned char raw[RAW];  // the next tokens' q, k and decay logits as they lie in memory
    __shared__ __align__(8) float s_all[DK];
    __shared__ int s_odd;  // MODE 0: a key or value up to here was no number
    const int colblocks = (dv + kCkCols - 1) / kCkCols;
    const int s = blockIdx.x, head = blockIdx.y / colblocks, col0 = (blockIdx.y % colblocks) * kCkCols, c = blockIdx.z;
    const int seq_first = seq_info[s * 4 + 0], seq_count = seq_info[s * 4 + 1], start = seq_info[s * 4 + 2], slot = seq_info[s * 4 + 3];
    int lo, hi, nseg;
    if (!la_segment(start, seq_count, c, lo, hi, nseg) || (MODE == 0 && c == nseg - 1)) return;
    const int first = seq_first + (lo - start), count = hi - lo;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int wcol = col0 + warp * 32;
    const bool live = wcol < dv;  // dv is a multiple of 32
    const bool slot_ok = slot >= 0 && slot < num_slots;
    float *const mine = state + (size_t)(slot_ok ? slot : 0) * slot_stride + (size_t)head * DK * dv;
    float *const seg = seg_state + (((size_t)s * max_segments + c) * heads + head) * DK * dv;

    float S[2][NT][4];
    {
        // the slot of a sequence that is cut is read in the launches before this one only: here the CTA of its last segment writes it
        const bool from_seg = MODE == 1 && nseg > 1, from_slot = !from_seg && c == 0 && lo > 0 && slot_ok;
        const float *const src = from_slot ? mine : seg;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    S[m][n][i] = live && (from_slot || from_seg) ? src[(size_t)(n * 8 + 2 * t + (i & 1)) * dv + wcol + m * 16 + g + (i & 2) * 4] : 0.f;
    }

    // a thread stages channels d0 .. of token j and 16 columns of v
    const int j = threadIdx.x >> 3, d0 = (threadIdx.x & 7) * PER, v0 = (threadIdx.x & 7) * 16;
    float bias[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) bias[i] = z_bias ? to_f(z_bias[(size_t)head * DK + d0 + i]) : 0.f;
    struct __align__(2 * PER) Row {
        bf16 x[PER];
    };
    const auto copy = [](void *to, const void *from, int bytes) {
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(to));
        if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(from) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(from) : "memory");
    };
    auto fetch = [&](int t0, int b) {  // a thread copies what it reads itself later, and v
        if (t0 + j < count) {
            const size_t tok = (size_t)(first + t0 + j);
            if (MODE) copy(raw + RAW_Q + (j * DK + d0) * 2, q + tok * q_token + (size_t)head * q_head + d0, 2 * PER);
            copy(raw + RAW_K + (j * DK + d0) * 2, k + tok * k_token + (size_t)head * k_head + d0, 2 * PER);
#pragma unroll
            for (int i = 0; i < PER; i += 4) copy(raw + RAW_Z + (j * DK + d0 + i) * 4, z + tok * z_token + (size_t)head * DK + d0 + i, 16);
#pragma unroll
            for (int i = 0; i < 16; i += 8)
                if (col0 + v0 + i < dv) copy(&s_v[b][j][v0 + i], v + tok * v_token + (size_t)head * v_head + col0 + v0 + i, 16);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 16; i += 8)  // columns that are not there
            if (col0 + v0 + i >= dv) *reinterpret_cast<uint4 *>(&s_v[b][j][v0 + i]) = make_uint4(0u, 0u, 0u, 0u);
    if (!MODE && threadIdx.x == 0) s_odd = 0;
    float total = 1.f;  // threads below DK: the segment's decay of their channel
    fetch(0, 0);
    for (int t0 = 0, b = 0; t0 < count; t0 += kCkTokens, b ^= 1) {
        const int n_tok = min(kCkTokens, count - t0);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        {  // past the last token: decay 1, key, query and value 0
            const bool in = j < n_tok;
            const float *const rz = reinterpret_cast<const float *>(raw + RAW_Z) + j * DK + d0;
            const Row rk = *reinterpret_cast<const Row *>(raw + RAW_K + (j * DK + d0) * 2);
            float a[PER], x[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const float zz = rz[i] + bias[i];
                a[i] = !in ? 1.f : decay_kind == 2 ? expf(-expf(zz)) : expf(log_sigmoid(zz) * inv_tau);
                x[i] = in ? to_f(rk.x[i]) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < PER; i += 4) {
                *reinterpret_cast<float4 *>(&s_alpha[j][d0 + i]) = make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
                *reinterpret_cast<float4 *>(&s_k[j][d0 + i]) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
            }
            if (MODE) {
                const Row rq = *reinterpret_cast<const Row *>(raw + RAW_Q + (j * DK + d0) * 2);
#pragma unroll
                for (int i = 0; i < PER; ++i) x[i] = in ? to_f(rq.x[i]) * q_scale : 0.f;
#pragma unroll
                for (int i = 0; i < PER; i += 4) *reinterpret_cast<float4 *>(&s_q[j][d0 + i]) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
            }
            if (!in)
#pragma unroll
                for (int i = 0; i < 16; i += 8) *reinterpret_cast<uint4 *>(&s_v[b][j][v0 + i]) = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        if (t0 + kCkTokens < count) fetch(t0 + kCkTokens, b ^ 1);
        // ---- q A and k R as terms: a thread a pair of channels and eight of the tokens, forward or backward (MODE 0: backward alone)
        if (lane < DK / 2 && (MODE || warp < 2)) {
            const int d = 2 * lane, back = MODE ? warp >> 1 : 1, late = warp & 1;  // late: behind the eight tokens of the other
            float2 a = make_float2(1.f, 1.f);
            if (late)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 x = *reinterpret_cast<const float2 *>(&s_alpha[back ? 15 - i : i][d]);
                    a.x *= x.x, a.y *= x.y;
                }
            const float(*const from)[DK] = back ? s_k : s_q;
            bf16(*const to)[kCkTokens][ROW] = back ? t_k : t_q;
#pragma unroll
            for (int i0 = 0; i0 < 8; ++i0) {
                const int i = back ? 15 - late * 8 - i0 : late * 8 + i0;
                const float2 x = *reinterpret_cast<const float2 *>(&s_alpha[i][d]), y = *reinterpret_cast<const float2 *>(&from[i][d]);
                if (!back) a.x *= x.x, a.y *= x.y;
                uint32_t term[3];
                ck_split(y.x * a.x, y.y * a.y, term);
#pragma unroll
                for (int u = 0; u < 3; ++u) *reinterpret_cast<uint32_t *>(&to[u][i][d]) = term[u];
                if (back) a.x *= x.x, a.y *= x.y;
            }
            if (back && late) *reinterpret_cast<float2 *>(&s_all[d]) = a;
        }
        if (!MODE && warp >= 2) {  // the idle warps: is every key and value a number?
            float test = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = ((warp - 2) * 32 + lane) * 4 + i;  // 16 bytes
                const uint4 x = *reinterpret_cast<const uint4 *>(&s_v[b][e >> 4][(e & 15) * 8]);
                const float2 x0 = tl::unpack2<bf16>(x.x), x1 = tl::unpack2<bf16>(x.y), x2 = tl::unpack2<bf16>(x.z), x3 = tl::unpack2<bf16>(x.w);
                test = fmaf((x0.x + x0.y) + (x1.x + x1.y) + ((x2.x + x2.y) + (x3.x + x3.y)), 0.f, test);
            }
#pragma unroll
            for (int e = (warp - 2) * 32 + lane; e < kCkTokens * DK / 2; e += 64) {
                const float2 x = *reinterpret_cast<const float2 *>(&s_k[0][0] + 2 * e);
                test = fmaf(x.x + x.y, 0.f, test);
            }
            if (test != 0.f) s_odd = 1;
        }
        // ---- P: sixteen lanes a token s, a warp two early and two late ones, so that all warps have as many steps
        if (MODE) {
            constexpr int CH = DK / 16;
            const int dc = (lane & 15) * CH;
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
                const int s0 = part ? 14 - 2 * warp : 2 * warp, ps = s0 + (lane >> 4), from = s0 & ~3;
                float r[CH];
#pragma unroll
                for (int i = 0; i < CH; ++i) r[i] = s_k[ps][dc + i];
#pragma unroll 1
                for (int t4 = from; t4 < kCkTokens; t4 += 4) {  // four tokens t, whose sums over the sixteen lanes end in four of these
                    float y[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        y[i] = 0.f;
#pragma unroll
                        for (int n = 0; n < CH; n += 2) {
                            const float2 x = *reinterpret_cast<const float2 *>(&s_alpha[t4 + i][dc + n]), w = *reinterpret_cast<const float2 *>(&s_q[t4 + i][dc + n]);
                            if (t4 + i > ps) r[n] *= x.x, r[n + 1] *= x.y;
                            y[i] = fmaf(w.x, r[n], y[i]), y[i] = fmaf(w.y, r[n + 1], y[i]);
                        }
                    }
                    const bool b3 = lane & 8, b2 = lane & 4;
                    const float u0 = (b3 ? y[2] : y[0]) + __shfl_xor_sync(0xffffffffu, b3 ? y[0] : y[2], 8);
                    const float u1 = (b3 ? y[3] : y[1]) + __shfl_xor_sync(0xffffffffu, b3 ? y[1] : y[3], 8);
                    float sum = (b2 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b2 ? u0 : u1, 4);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    const int tt = t4 + (b3 ? 2 : 0) + (b2 ? 1 : 0);
                    if ((lane & 3) == 0) {
                        uint32_t term[3];
                        ck_split(tt >= ps ? sum : 0.f, 0.f, term);
#pragma unroll
                        for (int u = 0; u < 3; ++u) *reinterpret_cast<unsigned short *>(&t_p[u][tt][ps]) = static_cast<unsigned short>(term[u]);
                    }
                }
                for (int e = lane; e < 2 * 3 * from; e += 32) t_p[e / 2 / from][e / 2 % from][s0 + (e & 1)] = from_f<bf16>(0.f);  // tokens before s
            }
        }
        __syncthreads();
        const auto step = [&](float (&x)[4], int tt, int n, float v0, float v8) {  // one token's step of channels n * 8 + 2t, + 1 and two columns
            const float2 decay = *reinterpret_cast<const float2 *>(&s_alpha[tt][n * 8 + 2 * t]), key = *reinterpret_cast<const float2 *>(&s_k[tt][n * 8 + 2 * t]);
            x[0] = fmaf(decay.x, x[0], key.x * v0), x[1] = fmaf(decay.y, x[1], key.y * v0);
            x[2] = fmaf(decay.x, x[2], key.x * v8), x[3] = fmaf(decay.y, x[3], key.y * v8);
        };
        bool walked[2] = {false, false};
        uint32_t va[2][4];  // v^T: 16 columns x 16 tokens
#pragma unroll
        for (int m = 0; m < 2; ++m) ck_ldm_t(va[m], &s_v[b][(lane & 7) + (lane >> 4) * 8][warp * 32 + m * 16 + (lane >> 3 & 1) * 8]);
        if (MODE) {
            const int row = (lane & 7) + (lane >> 4) * 8, half = (lane >> 3 & 1) * 8;  // B operands: tokens 0-7 | 8-15 x the two halves of 16
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                float o[2][4] = {}, low[2][4] = {};  // low: the products of all terms but the first two
                const auto add = [](float (&to)[4], const float (&x)[4]) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) to[i] += x[i];
                };
#pragma unroll
                for (int kk = 0; kk < KT; ++kk) {
                    uint32_t w[3][4], a[3][4], term[3];
#pragma unroll
                    for (int u = 0; u < 3; ++u) ck_ldm(w[u], &t_q[u][row][kk * 16 + half]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        ck_split(S[m][2 * kk + (i >> 1)][(i & 1) * 2], S[m][2 * kk + (i >> 1)][(i & 1) * 2 + 1], term);
#pragma unroll
                        for (int u = 0; u < 3; ++u) a[u][i] = term[u];
                    }
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
#pragma unroll
                        for (int sum = 2; sum >= 1; --sum)
#pragma unroll
                            for (int u = 0; u <= sum; ++u) ck_mma(low[n], a[u], w[sum - u][2 * n], w[sum - u][2 * n + 1]);
                        float high[4] = {};
                        ck_mma(high, a[0], w[0][2 * n], w[0][2 * n + 1]);
                        add(o[n], high);
                    }
                }
                float high[2][4] = {}, test = 0.f;
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    uint32_t w[4];
                    ck_ldm(w, &t_p[u == 0 ? 0 : 3 - u][row][half]);
#pragma unroll
                    for (int n = 0; n < 2; ++n) ck_mma(u == 0 ? high[n] : low[n], va[m], w[2 * n], w[2 * n + 1]);
                }
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    add(o[n], high[n]), add(o[n], low[n]);
                    test += (o[n][0] + o[n][1]) + (o[n][2] + o[n][3]);
                }
                float *const to = out + ((size_t)(first + t0) * heads + head) * dv + wcol + m * 16 + g;
                walked[m] = __any_sync(0xffffffffu, test - test != 0.f);
                if (walked[m]) {  // something is no number (an infinity's terms are infinity, NaN, NaN, and zero times it is NaN): token by token
#pragma unroll 1
                    for (int tt = 0; tt < n_tok; ++tt) {
                        const float v0 = to_f(s_v[b][tt][warp * 32 + m * 16 + g]), v8 = to_f(s_v[b][tt][warp * 32 + m * 16 + g + 8]);
                        float y0 = 0.f, y8 = 0.f;
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            step(S[m][n], tt, n, v0, v8);
                            const float2 x = *reinterpret_cast<const float2 *>(&s_q[tt][n * 8 + 2 * t]);
                            y0 = fmaf(x.x, S[m][n][0], fmaf(x.y, S[m][n][1], y0)), y8 = fmaf(x.x, S[m][n][2], fmaf(x.y, S[m][n][3], y8));
                        }
#pragma unroll
                        for (int i = 1; i < 4; i <<= 1) y0 += __shfl_xor_sync(0xffffffffu, y0, i), y8 += __shfl_xor_sync(0xffffffffu, y8, i);
                        if (live && t == 0) to[(size_t)tt * heads * dv] = y0, to[(size_t)tt * heads * dv + 8] = y8;
                    }
                } else if (live) {
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int tt = n * 8 + 2 * t + (i & 1);
                            if (tt < n_tok) to[(size_t)tt * heads * dv + (i & 2) * 4] = o[n][i];
                        }
                }
            }
        }
        // ---- S^T <- S^T diag(A_16) + v^T (k R)
        if (MODE ? walked[0] || walked[1] : s_odd != 0) {
#pragma unroll
            for (int m = 0; m < 2; ++m)
                if (!walked[m])
#pragma unroll 1
                    for (int tt = 0; tt < n_tok; ++tt) {
                        const float v0 = to_f(s_v[b][tt][warp * 32 + m * 16 + g]), v8 = to_f(s_v[b][tt][warp * 32 + m * 16 + g + 8]);
#pragma unroll
                        for (int n = 0; n < NT; ++n) step(S[m][n], tt, n, v0, v8);
                    }
        } else {
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                float more[2][2][4] = {};
#pragma unroll
                for (int u = 2; u >= 0; --u) {
                    uint32_t w[4];
                    ck_ldm_t(w, &t_k[u][(lane & 7) + (lane >> 3 & 1) * 8][n * 8 + (lane >> 4) * 8]);
#pragma unroll
                    for (int m = 0; m < 2; ++m) ck_mma(more[m][0], va[m], w[0], w[1]), ck_mma(more[m][1], va[m], w[2], w[3]);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = *reinterpret_cast<const float2 *>(&s_all[(n + h) * 8 + 2 * t]);
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int i = 0; i < 4; ++i) S[m][n + h][i] = fmaf(i & 1 ? x.y : x.x, S[m][n + h][i], more[m][h][i]);
                }
            }
        }
        if (MODE == 0 && threadIdx.x < DK) total *= s_all[threadIdx.x];
    }
    float *const dst = MODE == 0 ? seg : c == nseg - 1 && slot_ok ? mine : nullptr;
    if (dst != nullptr && live) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) dst[(size_t)(n * 8 + 2 * t + (i & 1)) * dv + wcol + m * 16 + g + (i & 2) * 4] = S[m][n][i];
    }
    if (MODE == 0 && col0 == 0 && threadIdx.x < DK) seg_decay[(((size_t)s * max_segments + c) * heads + head) * DK + threadIdx.x] = total;
}

// The segments' start states where their end states were, in order: start[0] the sequence's own state (its slot's, or zero), start[1] = end[0] (that
// segment began from it), start[c + 1] = decay[c] start[c] + end[c].  A thread four neighbouring columns of a row; eight segments' numbers are on their way at once.
__global__ void __launch_bounds__(256)
decay_starts_kernel(const int32_t *__restrict__ seq_info, int heads, int dk, int dv, int max_segments, float *__restrict__ seg_state, const float *__restrict__ seg_decay,
                    const float *__restrict__ state, long long slot_stride, int num_slots) {
    const int s = blockIdx.x, head = blockIdx.y, e = (blockIdx.z * blockDim.x + threadIdx.x) * 4;
    int lo, hi, nseg;
    const int start = seq_info[s * 4 + 2], slot = seq_info[s * 4 + 3];
    la_segment(start, seq_info[s * 4 + 1], 0, lo, hi, nseg);
    if (nseg <= 1 || e >= dk * dv) return;
    constexpr int kAhead = 8;
    float4 own = make_float4(0.f, 0.f, 0.f, 0.f);
    if (start > 0 && slot >= 0 && slot < num_slots) {
        const float *const mine = state + (size_t)slot * slot_stride + (size_t)head * dk * dv + e;
        own = make_float4(mine[0], mine[1], mine[2], mine[3]);
    }
    float *seg = seg_state + ((size_t)s * max_segments * heads + head) * dk * dv + e;
    const float *dec = seg_decay + ((size_t)s * max_segments * heads + head) * dk + e / dv;
    const size_t seg_step = (size_t)heads * dk * dv, dec_step = (size_t)heads * dk;
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c0 = 0; c0 < nseg; c0 += kAhead, seg += kAhead * seg_step, dec += kAhead * dec_step) {
        float4 end[kAhead];
        float decay[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (c0 + u + 1 < nseg) end[u] = *reinterpret_cast<const float4 *>(seg + u * seg_step), decay[u] = dec[u * dec_step];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (c0 + u < nseg) {
                *reinterpret_cast<float4 *>(seg + u * seg_step) = c0 + u == 0 ? own : S;
                if (c0 + u + 1 < nseg) {
                    const float d = decay[u];
                    S = make_float4(fmaf(d, S.x, end[u].x), fmaf(d, S.y, end[u].y), fmaf(d, S.z, end[u].z), fmaf(d, S.w, end[u].w));
                }
            }
    }
}

// out[t, h, :] = o[t, h, :] / rms(o[t, h, :]) * w * act(gate[t, h, :]); one warp per (token, head).  act 0 = none, 1 = silu,
// 2 = sigmoid; w == NULL: no weight; wide_weight: w is [heads * dv] (every head its own part) instead of [dv] shared by the
// heads; gate_first: the gate multiplies o BEFORE the norm, out = n / rms(n) * w with n = o * act(gate).  floor: a row of o has one
// more column, and o is first divided by max(|that column|, floor[t, h]) + den_eps (a normalised memory's read-out).
template <typename T>
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float *__restrict__ o, const T *__restrict__ w, float eps, const T *__restrict__ gate, long long g_token, int act,
                      T *__restrict__ out, long long rows, int heads, int dv, int wide_weight, int gate_first, int o_row,
                      const float *__restrict__ floor, float den_eps) {
    long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const long long t = row / heads;
    const int head = (int)(row - t * heads);
    const float *src = o + (size_t)row * o_row;
    const float share = floor ? 1.0f / (fmaxf(fabsf(src[dv]), floor[row]) + den_eps) : 1.f;
    auto gated = [&](int d) {
        float gv = to_f(gate[(size_t)t * g_token + (size_t)head * dv + d]);
        return act == 1 ? gv / (1.0f + expf(-gv)) : act == 2 ? 1.0f / (1.0f + expf(-gv)) : gv;
    };
    const bool first = gate && gate_first;
    float ss = 0.f;
    for (int d = lane; d < dv; d += 32) {
        float x = first ? src[d] * gated(d) : src[d] * share;
        ss += x * x;
    }
    ss = warp_sum(ss);
    float inv = 1.0f / sqrtf(ss / (float)dv + eps);
    const T *wr = w ? w + (wide_weight ? (size_t)head * dv : 0) : nullptr;
    for (int d = lane; d < dv; d += 32) {
        float y = src[d] * share * inv * (wr ? to_f(wr[d]) : 1.f);
        if (gate) y *= gated(d);
        out[(size_t)row * dv + d] = from_f<T>(y);
    }
}

// The same for rows of whole fours (16 bytes of o, 8 of a bf16 gate an access) and at most PIECES times 128 columns: a row's numbers are requested
// together and kept, where the kernel above makes three round trips of 4-byte accesses (2048 tokens of 16 heads of 128 columns: 18 -> 12.6 us, now bound by
// the exponentials and divisions).
template <typename T, int PIECES>
__global__ void __launch_bounds__(256)
head_norm_gate_wide_kernel(const float *__restrict__ o, const T *__restrict__ w, float eps, const T *__restrict__ gate, long long g_token, int act,
                           T *__restrict__ out, long long rows, int heads, int dv, int wide_weight, int gate_first, int o_row,
                           const float *__restrict__ floor, float den_eps) {
    const unsigned row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // below 2^31 (a division of 64 bits is a hundred instructions)
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const unsigned t = row / (unsigned)heads;
    const int head = (int)(row - t * heads);
    const float *src = o + (size_t)row * o_row;
    const T *wr = w ? w + (wide_weight ? (size_t)head * dv : 0) : nullptr;
    const T *gr = gate ? gate + (size_t)t * g_token + (size_t)head * dv : nullptr;
    struct __align__(4 * sizeof(T)) Four {
        T v[4];
    };
    float4 x[PIECES];
    Four g[PIECES], k[PIECES];
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int d = (i * 32 + lane) * 4;
        x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (d >= dv) continue;
        x[i] = *reinterpret_cast<const float4 *>(src + d);
        if (gr) g[i] = *reinterpret_cast<const Four *>(gr + d);
        if (wr) k[i] = *reinterpret_cast<const Four *>(wr + d);
    }
    const float share = floor ? 1.0f / (fmaxf(fabsf(src[dv]), floor[row]) + den_eps) : 1.f;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        float *const v = &x[i].x;
        const bool in = (i * 32 + lane) * 4 < dv;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float a = 1.f;
            if (gr && in) {
                const float gv = to_f(g[i].v[j]);
                a = act == 1 ? gv / (1.0f + expf(-gv)) : act == 2 ? 1.0f / (1.0f + expf(-gv)) : gv;
            }
            v[j] *= share;
            const float y = gate_first ? v[j] * a : v[j];
            if (in) ss += y * y;
            v[j] *= a;  // what is left is the norm and its weight
        }
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dv + eps);
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int d = (i * 32 + lane) * 4;
        if (d >= dv) continue;
        const float *const v = &x[i].x;
        Four y;
#pragma unroll
        for (int j = 0; j < 4; ++j) y.v[j] = from_f<T>(v[j] * inv * (wr ? to_f(k[i].v[j]) : 1.f));
        *reinterpret_cast<Four *>(out + (size_t)row * dv + d) = y;
    }
}

}  // namespace tlb

using namespace tlb;

extern "C" {

size_t tlb_decay_scan_workspace(int tokens, int num_seqs, int max_tokens_per_seq, int heads, int dk, int dv) {
    if (max_tokens_per_seq <= kLaSegment) return 0;
    size_t segs = (size_t)num_seqs * (2 + (max_tokens_per_seq - 1) / kLaSegment);
    return (segs * heads * ((size_t)dk * dv + dk) + ((size_t)tokens + 2 * kLaSegment * (size_t)num_seqs) * heads * dk + 1) * sizeof(float);
}

int tlb_decay_scan(const void *q, long long q_token, long long q_head, const void *k, long long k_token, long long k_head, const void *v,
                   long long v_token, long long v_head, const float *z, long long z_token, const void *z_bias, float tau, const float *head_decay,
                   const float *rope_cos, const float *rope_sin, int rope_dims, int rope_interleaved, float q_scale, int heads,
                   int dk, int dv, const int32_t *seq_info, int num_seqs, int tokens, int max_tokens_per_seq, float *state, long long slot_stride, int num_slots,
                   float *out, void *workspace, size_t workspace_bytes, int decay_kind, const void *a_log, const void *bonus, int qk_heads,
                   const void *skip, int v_cols, int dtype, void *stream) {
    if (num_seqs <= 0) return TL_OK;
    if (qk_heads <= 0) qk_heads = heads;
    if ((decay_kind != 0 && decay_kind != 2 && decay_kind != 3 && decay_kind != 4) || (decay_kind != 0 && (!z || head_decay)) || (decay_kind == 3 && !a_log) ||
        (decay_kind == 4 && ((uintptr_t)z % 8 || z_token % 2)) || heads % qk_heads)
        return tl::fail(TL_EINVAL, "decay_scan: bad decay kind or head groups");
    if (v_cols <= 0) v_cols = dv;
    if (v_cols > dv) return tl::fail(TL_EINVAL, "decay_scan: %d value columns in a state of %d", v_cols, dv);
    if (!q || !k || !v || (!z && !head_decay) || !seq_info || !state || !out || heads <= 0 || dk <= 0 || dv <= 0 || (z && !(tau > 0.f)) ||
        num_slots <= 0 || max_tokens_per_seq <= 0)
        return tl::fail(TL_EINVAL, "decay_scan: bad argument");
    if (rope_dims < 0 || (rope_dims & 1) || rope_dims > dk || (rope_dims > 0 && (!rope_cos || !rope_sin)))
        return tl::fail(TL_EINVAL, "decay_scan: bad rotation of %d of %d entries", rope_dims, dk);
    if (dk > 256) return tl::fail(TL_EINVAL, "decay_scan: key size %d > 256", dk);
    // portions longer than a segment are cut at absolute multiples of the segment length and run in three passes
    const bool segmented = max_tokens_per_seq > kLaSegment;
    const int max_segments = segmented ? 2 + (max_tokens_per_seq - 1) / kLaSegment : 1;
    float *seg_state = nullptr, *seg_decay = nullptr, *decayed = nullptr;
    float2 *last_steps = nullptr;
    if (segmented) {
        if (!workspace || workspace_bytes < tlb_decay_scan_workspace(tokens, num_seqs, max_tokens_per_seq, heads, dk, dv))
            return tl::fail(TL_EWORKSPACE, "decay_scan: workspace missing or too small");
        seg_state = (float *)workspace;
        seg_decay = seg_state + (size_t)num_seqs * max_segments * heads * dk * dv;
        decayed = seg_decay + (size_t)num_seqs * max_segments * heads * dk;
        float *end = decayed + (size_t)tokens * heads * dk;
        last_steps = (float2 *)(end + ((uintptr_t)end / 4 & 1));  // 8-byte aligned
    }
    const bool scalar = head_decay || decay_kind >= 3;
    if (scalar && bonus) return tl::fail(TL_EINVAL, "decay_scan: a bonus goes with a decay per key channel");
    cudaStream_t st = as_stream(stream);
    const int kr = ceil_div(dk, kLaLanes);
    // Four, two or one columns a thread (64 registers of state): more read a row's staged numbers fewer times, fewer give more CTAs
    // to hide the staging behind (16 heads, 33 segments: 191 us for both launches of the scan with four, 217 with two; 8 heads: 154
    // and 117).  A step of few tokens takes one, so that more CTAs share the state's traffic.
    const auto ctas = [&](int nc) { return (long long)heads * ceil_div(dv, kLaThreads / kLaLanes * nc) * num_seqs * max_segments; };
    int nc = 1;
    for (int more = kr <= 16 ? 4 : kr <= 32 ? 2 : 1; more > 1 && max_tokens_per_seq > 4 && nc == 1; more /= 2)
        if (ctas(more) >= 3LL * sm_count()) nc = more;
#define TLB_DS_N(KRV, PASS, GZ, BON, SCA, NCV)                                                                                                           \
    decay_scan_kernel<T, KRV, (KRV > 32 ? 8 : 16), BON, SCA, NCV, PASS != 0><<<dim3(num_seqs, heads * ceil_div(dv, kLaThreads / kLaLanes * NCV), GZ), kLaThreads, 0, st>>>(  \
        (const T *)q, q_token, q_head, (const T *)k, k_token, k_head, (const T *)v, v_token, v_head, z, z_token, (const T *)z_bias, z ? 1.0f / tau : 0.f, head_decay, \
        rope_cos, rope_sin, rope_dims, rope_interleaved, q_scale, heads, dk, dv, seq_info, state, slot_stride, num_slots, out, max_segments, seg_state, seg_decay, \
        decayed, last_steps, decay_kind, (const T *)a_log, (const T *)bonus, qk_heads, (const T *)skip, v_cols)
#define TLB_DS_B(KRV, PASS, GZ, BON, SCA)                                                                     \
    do {                                                                                                      \
        if (KRV <= 16 && nc == 4) TLB_DS_N(KRV, PASS, GZ, BON, SCA, (KRV <= 16 ? 4 : 1));                      \
        else if (KRV <= 32 && nc == 2) TLB_DS_N(KRV, PASS, GZ, BON, SCA, (KRV <= 32 ? 2 : 1));                 \
        else TLB_DS_N(KRV, PASS, GZ, BON, SCA, 1);                                                            \
    } while (0)
#define TLB_DS_K(KRV, PASS, GZ) do { if (bonus) TLB_DS_B(KRV, PASS, GZ, true, false); else if (scalar) TLB_DS_B(KRV, PASS, GZ, false, true); else TLB_DS_B(KRV, PASS, GZ, false, false); } while (0)
#define TLB_DS(PASS, GZ) TLB_DISPATCH(dtype, "decay_scan", if (kr <= 8) TLB_DS_K(8, PASS, GZ); else if (kr <= 16) TLB_DS_K(16, PASS, GZ); else if (kr <= 32) TLB_DS_K(32, PASS, GZ); else TLB_DS_K(64, PASS, GZ))
    if (!segmented) {
        TLB_DS(0, 1);
        TL_LAUNCH_CHECK("decay_scan");
        return TL_OK;
    }
    // the tensor cores' form: a decay per key channel from logits, bf16, whole 16-byte rows; the rest (rotation, bonus, skip, a normaliser, grouped
    // heads, other sizes) walks
    const auto rows16 = [](const void *p, long long token, long long head) { return (uintptr_t)p % 16 == 0 && token % 8 == 0 && head % 8 == 0; };
    if (dtype == TL_BF16 && !scalar && !bonus && !skip && rope_dims == 0 && qk_heads == heads && v_cols == dv && (dk == 32 || dk == 64) && dv % 32 == 0 &&
        rows16(q, q_token, q_head) && rows16(k, k_token, k_head) && rows16(v, v_token, v_head) && tl::aligned16(z) && z_token % 4 == 0 && tl::aligned16(workspace)) {
        const dim3 grid(num_seqs, heads * ceil_div(dv, kCkCols), max_segments);
#define TLB_CHUNK(DKV, MODE)                                                                                                                                    \
    decay_chunk_kernel<DKV, MODE><<<grid, 128, 0, st>>>((const bf16 *)q, q_token, q_head, (const bf16 *)k, k_token, k_head, (const bf16 *)v, v_token, v_head, z, \
                                                        z_token, (const bf16 *)z_bias, 1.0f / tau, q_scale, heads, dv, seq_info, state, slot_stride, num_slots,  \
                                                        out, max_segments, seg_state, seg_decay, decay_kind)
        if (dk == 64) TLB_CHUNK(64, 0); else TLB_CHUNK(32, 0);
        TL_LAUNCH_CHECK("decay_scan (end states)");
        decay_starts_kernel<<<dim3(num_seqs, heads, ceil_div(dk * dv, 1024)), 256, 0, st>>>(seq_info, heads, dk, dv, max_segments, seg_state, seg_decay,
                                                                                                 state, slot_stride, num_slots);
        TL_LAUNCH_CHECK("decay_scan (start states)");
        if (dk == 64) TLB_CHUNK(64, 1); else TLB_CHUNK(32, 1);
        TL_LAUNCH_CHECK("decay_scan (outputs)");
#undef TLB_CHUNK
        return TL_OK;
    }
    TLB_DS(1, max_segments);
    TL_LAUNCH_CHECK("decay_scan (segments)");
    const bool vec = dk % 4 == 0 && dv % 4 == 0 && tl::aligned16(workspace) && tl::aligned16(out);
#define TLB_COMBINE(W)                                                                                                                          \
    decay_combine_kernel<T, W><<<dim3(num_seqs, heads, ceil_div(dk * dv, 256 * W)), 256, 0, st>>>(seq_info, state, slot_stride, num_slots, heads, dk, dv, max_segments, \
                                                                                                 seg_state, seg_decay, last_steps, (const T *)v, v_token, v_head, v_cols)
    TLB_DISPATCH(dtype, "decay_scan", if (vec) TLB_COMBINE(4); else TLB_COMBINE(1));
#undef TLB_COMBINE
    TL_LAUNCH_CHECK("decay_scan (combine)");
    const dim3 og(num_seqs, heads * ceil_div(dv, kLaOutCols), max_segments - 1);
    if (vec) decay_output_kernel<true><<<og, 128, 0, st>>>(seq_info, heads, dk, dv, max_segments, seg_state, decayed, out);
    else decay_output_kernel<false><<<og, 128, 0, st>>>(seq_info, heads, dk, dv, max_segments, seg_state, decayed, out);
    TL_LAUNCH_CHECK("decay_scan (outputs)");
#undef TLB_DS
#undef TLB_DS_K
#undef TLB_DS_B
#undef TLB_DS_N
    return TL_OK;
}

int tlb_head_norm_gate(const float *o, const void *w, float eps, const void *gate, long long g_token, int act, void *out, int tokens, int heads,
                       int dv, int wide_weight, int gate_first, int o_row, const float *floor, float den_eps, int dtype, void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!o || !out || heads <= 0 || dv <= 0 || act < 0 || act > 2) return tl::fail(TL_EINVAL, "head_norm_gate: bad argument");
    if (o_row <= 0) o_row = dv;
    if (o_row < dv + (floor ? 1 : 0) || (floor && gate_first)) return tl::fail(TL_EINVAL, "head_norm_gate: bad row or normaliser");
    long long rows = (long long)tokens * heads;
    const size_t four = dtype == TL_BF16 ? 8 : 16;
    const auto fits = [&](const void *p) { return p == nullptr || (uintptr_t)p % four == 0; };
    if (rows < (1ll << 31) && dv % 4 == 0 && dv <= 512 && o_row % 4 == 0 && g_token % 4 == 0 && tl::aligned16(o) && fits(w) && fits(gate) && fits(out)) {
        const unsigned ctas = (unsigned)((rows + 7) / 8);
#define TLB_WIDE(P)                                                                                                                                          \
    head_norm_gate_wide_kernel<T, P><<<ctas, 256, 0, as_stream(stream)>>>(o, (const T *)w, eps, (const T *)gate, g_token, act, (T *)out, rows, heads, dv, \
                                                                          wide_weight, gate_first, o_row, floor, den_eps)
        TLB_DISPATCH(dtype, "head_norm_gate", if (dv <= 128) TLB_WIDE(1); else if (dv <= 256) TLB_WIDE(2); else TLB_WIDE(4));
#undef TLB_WIDE
        TL_LAUNCH_CHECK("head_norm_gate");
        return TL_OK;
    }
    TLB_DISPATCH(dtype, "head_norm_gate",
                 head_norm_gate_kernel<T><<<(unsigned)((rows + 3) / 4), 128, 0, as_stream(stream)>>>(o, (const T *)w, eps, (const T *)gate, g_token, act,
                                                                                                    (T *)out, rows, heads, dv, wide_weight, gate_first, o_row, floor, den_eps));
    TL_LAUNCH_CHECK("head_norm_gate");
    return TL_OK;
}

}  // extern "C"
