// WKV state recurrences of RWKV v5 / v6 / v7 for sm_100a.
//
// Replaces time_mix_v5.wgsl, time_mix_v6.wgsl and time_mix_v7.wgsl.  The reference runs one
// dispatch with C/4 threads that is serial over every token of the job and round-trips the whole
// S x S state through global memory on each token.  Here a CTA owns a share of the columns of one (sequence, head) pair and
// keeps them in registers for the sequence's whole run of tokens; the per-token vectors shared by the head (k, r, w, ...)
// reach shared memory a chunk ahead, and the state touches HBM once on the way in and once on the way out.  Sequences,
// heads and columns are independent, so the grid is (heads x shares of the columns, batch slots).
//
// State layout (reference: src/runtime/v6.rs:187-197): f32 view [C, S+1, B]; row 0 = token-shift
// carry, row 1+i = key index i for all heads side by side (column h*S + j = value index j).
#include "device.cuh"
#include "launch.cuh"

namespace wrk {
namespace k {

namespace {

// Finds the contiguous run of tokens that belongs to batch slot `slot`.  Returns false when the
// slot has no token in this job.  `carry` (when given) receives 1 + the last token of the run whose cursor says it
// ends its sequence's part of the job (t - token + 1 == len), or 0 when there is none: the token whose layer input
// becomes the token-shift carry row.
struct RunScratch {
    uint32_t start, count, carry;
};
__device__ __forceinline__ bool find_run(const uint32_t* cursors, int wide, uint32_t T, uint32_t slot, RunScratch* sh,
                                         uint32_t& start, uint32_t& count, uint32_t* carry = nullptr) {
    if (threadIdx.x == 0) {
        sh->start = 0xffffffffu;
        sh->count = 0;
        sh->carry = 0;
    }
    __syncthreads();
    uint32_t my_min = 0xffffffffu, my_cnt = 0, my_carry = 0;
    for (uint32_t t = threadIdx.x; t < T; t += blockDim.x) {
        const CursorD c = cursor_at(cursors, wide, t);
        if (c.batch == slot) {
            my_min = min(my_min, t);
            ++my_cnt;
            if (t - c.token + 1u == c.len) my_carry = t + 1;
        }
    }
    if (my_cnt) {
        atomicMin(&sh->start, my_min);
        atomicAdd(&sh->count, my_cnt);
        if (my_carry) atomicMax(&sh->carry, my_carry);
    }
    __syncthreads();
    start = sh->start;
    count = sh->count;
    if (carry) *carry = sh->carry;
    return count != 0;
}

// Four consecutive channels from element i, a multiple of four.
__device__ __forceinline__ float4 load_quad(const void* base, int dtype, size_t i) {
    if (dtype != WRK_F16) return *reinterpret_cast<const float4*>(static_cast<const float*>(base) + i);
    const uint2 q = *reinterpret_cast<const uint2*>(static_cast<const __half*>(base) + i);
    const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&q.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 splat4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Sums N values per lane over G neighbouring lanes (both powers of two).  Every step halves the values a lane still carries
// and sends the other half to its partner: N - 1 shuffles instead of N log2 G.  Lane g of the G ends with the sums of values
// g N / G .. in y[0 ..] (N >= G), or with value g N / G (N < G).
template <int N, int G>
__device__ __forceinline__ void sum_scatter(float (&y)[N], uint32_t g) {
    int width = N;
#pragma unroll
    for (int mask = G / 2; mask >= 1; mask /= 2) {
        if (width > 1) {
            width /= 2;
            const bool upper = (g & mask) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i >= width) break;
                const float keep = upper ? y[i + width] : y[i], send = upper ? y[i] : y[i + width];
                y[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
            }
        } else {
            y[0] += __shfl_xor_sync(0xffffffffu, y[0], mask);
        }
    }
}

// v5 / v6.  The columns of a head's S x S state (rows = key index, columns = value index) do not depend on one another, so
// a CTA takes NC of them, for the sequence's whole run of tokens: 64 heads of 64 channels are 128 CTAs of 32 columns, one
// per SM.  A thread keeps a 4 x 4 tile of the state in registers, as pairs of rows (two products per instruction); the
// S / 4 row groups of a column group are lanes of one warp.  A token is tied to the one before it by one fma of the state
// alone; four tokens' outputs are summed over the row groups together (sum_scatter: 15 shuffles for 16 values).  The
// tokens' k, r, w and v rows reach shared memory a chunk of TC tokens at a time, loaded a chunk ahead into registers while
// the current chunk is computed (one barrier per chunk).  Past the run's end k, r, v are 0 and w is 1: such a token changes
// nothing.
// Measured at 64 heads of 64, one sequence: 35 us for 256 tokens and 0.12 us per further token.  A CTA per whole head
// took 95 us.  Tiles of
// 4 x 2 with twice the warps: 33 us, but 6 instead of 4 us for a single token.
template <int S, int NC>
__global__ void __launch_bounds__((S / 4) * (NC / 4)) time_mix_v56_kernel(const WkvArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int RG = S / 4, NT = RG * (NC / 4), CGW = 32 / RG, TC = S <= 64 ? 16 : 8, QT = (TC * RG + NT - 1) / NT;
    static_assert(RG == 8 || RG == 16 || RG == 32, "the row groups of a column group are lanes of one warp");
    enum { IN_K = 0, IN_R = 1, IN_W = 2 };
    __shared__ __align__(16) float sin[2][3][TC][S], sv[2][TC][NC];
    __shared__ RunScratch run;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t rg = lane % RG, cg = (tid >> 5) * CGW + lane / RG;  // rows 4 rg .., columns 4 cg .. of the CTA's
    const uint32_t h = blockIdx.x / (S / NC), part = blockIdx.x % (S / NC), slot = blockIdx.y, C = a.S * a.H, c0 = h * S;
    const uint32_t v0 = c0 + part * NC;  // the CTA's first column among all channels

    uint32_t start, count, carry;
    if (!find_run(a.cursors, a.wide, a.T, slot, &run, start, count, &carry)) return;
    // The token-shift carry row takes the layer input of the run's closing token.  Nothing in this kernel reads that
    // row, so it is written now, before the token's input is overwritten with its output; the token loop below then
    // has no cursor to look at and no branch.
    if (carry != 0) {
        for (uint32_t j = tid; j < NC; j += NT)
            static_cast<float*>(a.state.base)[a.state.index(v0 + j, 0, slot)] = dload(a.x, a.dtype, (size_t)(carry - 1) * C + v0 + j);
    }

    float2 st[2][4], u[2];  // st[pair of rows][column]
    float* state[4];
    bool vec = true;  // a view's rows may start anywhere
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        state[r] = static_cast<float*>(a.state.base) + a.state.index(v0 + 4 * cg, 1 + 4 * rg + r, slot);
        vec = vec && reinterpret_cast<uintptr_t>(state[r]) % 16 == 0;
    }
    auto load_row = [&](const float* p) { return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]); };
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        u[p] = make_float2(a.time_first[c0 + 4 * rg + 2 * p], a.time_first[c0 + 4 * rg + 2 * p + 1]);
        const float4 s0 = load_row(state[2 * p]), s1 = load_row(state[2 * p + 1]);
        st[p][0] = make_float2(s0.x, s1.x), st[p][1] = make_float2(s0.y, s1.y);
        st[p][2] = make_float2(s0.z, s1.z), st[p][3] = make_float2(s0.w, s1.w);
    }

    // staging: (token, four channels) pairs tid, tid + NT, ... of the TC RG pairs of a chunk
    float4 gk[QT], gr[QT], gw[QT], gv[QT];
    auto load_chunk = [&](uint32_t chunk) {
#pragma unroll
        for (int q = 0; q < QT; ++q) {
            const uint32_t idx = tid + q * NT, m = chunk * TC + idx / RG, c = 4 * (idx % RG);
            gk[q] = gr[q] = gv[q] = splat4(0.f);
            gw[q] = splat4(1.f);
            if (idx < TC * RG && m < count) {
                const size_t ti = (size_t)(start + m) * C;
                gk[q] = load_quad(a.k, a.dtype, ti + c0 + c);
                gr[q] = load_quad(a.r, a.dtype, ti + c0 + c);
                gw[q] = *reinterpret_cast<const float4*>(a.time_decay + (a.per_token_decay ? ti : 0) + c0 + c);
                if (c < NC) gv[q] = load_quad(a.v, a.dtype, ti + v0 + c);
            }
        }
    };
    auto store_chunk = [&](int buf) {
#pragma unroll
        for (int q = 0; q < QT; ++q) {
            const uint32_t idx = tid + q * NT, n = idx / RG, c = 4 * (idx % RG);
            if (idx < TC * RG) {
                *reinterpret_cast<float4*>(&sin[buf][IN_K][n][c]) = gk[q];
                *reinterpret_cast<float4*>(&sin[buf][IN_R][n][c]) = gr[q];
                *reinterpret_cast<float4*>(&sin[buf][IN_W][n][c]) = gw[q];
                if (c < NC) *reinterpret_cast<float4*>(&sv[buf][n][c]) = gv[q];
            }
        }
    };
    // four tokens, n0 .. of the chunk; the first of them is token t of the job, `left` of them exist
    auto tokens4 = [&](int buf, uint32_t n0, uint32_t t, uint32_t left) {
        float y[16];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const float4 kq = *reinterpret_cast<const float4*>(&sin[buf][IN_K][n0 + n][4 * rg]);
            const float4 rq = *reinterpret_cast<const float4*>(&sin[buf][IN_R][n0 + n][4 * rg]);
            const float4 wq = *reinterpret_cast<const float4*>(&sin[buf][IN_W][n0 + n][4 * rg]);
            const float4 vq = *reinterpret_cast<const float4*>(&sv[buf][n0 + n][4 * cg]);
            const float vc[4] = {vq.x, vq.y, vq.z, vq.w};
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const float2 v2 = make_float2(vc[cc], vc[cc]);
                const float2 kv0 = __fmul2_rn(lo2(kq), v2), kv1 = __fmul2_rn(hi2(kq), v2);
                const float2 y2 = __ffma2_rn(hi2(rq), __ffma2_rn(u[1], kv1, st[1][cc]), __fmul2_rn(lo2(rq), __ffma2_rn(u[0], kv0, st[0][cc])));
                st[0][cc] = __ffma2_rn(lo2(wq), st[0][cc], kv0);
                st[1][cc] = __ffma2_rn(hi2(wq), st[1][cc], kv1);
                y[4 * n + cc] = y2.x + y2.y;
            }
        }
        sum_scatter<16, RG>(y, rg);
        constexpr int OUT = RG <= 16 ? 16 / RG : 1;
#pragma unroll
        for (int e = 0; e < OUT; ++e) {
            const uint32_t i = rg * 16 / RG + e, n = i / 4;
            if ((RG <= 16 || (rg & 1) == 0) && n < left) dstore(a.x, a.dtype, (size_t)(t + n) * C + v0 + 4 * cg + i % 4, y[e]);
        }
    };
    const uint32_t chunks = (count + TC - 1) / TC;
    load_chunk(0);
    store_chunk(0);
    __syncthreads();

    for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
        const int buf = chunk & 1;
        const bool more = chunk + 1 < chunks;
        if (more) load_chunk(chunk + 1);  // in flight while this chunk's tokens are computed
        const uint32_t left = count - chunk * TC, t0 = start + chunk * TC;
        if (left >= TC) {
#pragma unroll
            for (uint32_t n = 0; n < TC; n += 4) tokens4(buf, n, t0 + n, 4);
        } else {
#pragma unroll 1
            for (uint32_t n = 0; n < left; n += 4) tokens4(buf, n, t0 + n, left - n);
        }
        if (more) store_chunk(buf ^ 1);  // last read during the previous chunk, before its closing barrier
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float2* s = st[r / 2];
        const float4 v = r % 2 == 0 ? make_float4(s[0].x, s[1].x, s[2].x, s[3].x) : make_float4(s[0].y, s[1].y, s[2].y, s[3].y);
        if (vec) *reinterpret_cast<float4*>(state[r]) = v;
        else state[r][0] = v.x, state[r][1] = v.y, state[r][2] = v.z, state[r][3] = v.w;
    }
}

// ---- v5 / v6 in blocks of 16 tokens ("chunk-parallel") ------------------------------------------------------------
// The recurrence  y_t = r_t . (u k_t v_t^T + S_(t-1)),  S_t = diag(w_t) S_(t-1) + k_t v_t^T  unrolled over a block of
// L = 16 tokens that starts from state S0 (rows i = key index, columns j = value index, per head):
//   y_t   = (r_t Pe_t) S0  +  sum_(s<=t) A[t][s] v_s,      S_end = diag(Pe_L) S0 + sum_s (k_s E_s) v_s^T
//   Pe_t  = prod_(m<t) w_m   (Pe_0 = 1),   E_s = prod_(m>s) w_m,
//   A[t][s] = sum_i r_t[i] k_s[i] prod_(s<m<t) w_m[i]  (s < t),   A[t][t] = sum_i r_t[i] u[i] k_t[i].
// Every product of decays is taken forwards (no division, nothing can overflow; what underflows is a contribution that
// has decayed to nothing).  The work of a block is then three small matrix products - [16 x 64][64 x 64] for the state's
// share of y, [16 x 16][16 x 64] for the block's own tokens and [64 x 16][16 x 64] for the new state - in which no
// element waits for another: 4 x 4 register tiles in fp32 on the CUDA cores, operands from shared memory.
// Two CTAs of 256 threads per (head of 64 channels, batch slot), each with 32 of the state's columns, which do not depend on one
// another (both form A and the decay products); the state tile of a thread stays in registers from block to block; the
// tokens' rows are staged a block ahead as in the serial kernel.  Every element is summed in the order that one CTA per head
// took, so its bits are the same.  256 tokens of 64 heads: 76 -> 68 us, and 53 (0.21 per token) with the loads of a block in flight
// together.  The serial kernel above has become the faster one (35 us, 0.14 per token); it sums in another order, and what that
// changes in the last bit of a state grows through the layers of a deep model (24 layers of random weights: to 1e-2 of the last
// layer's state).  It is also no further from float64 (256 tokens: outputs 8.8e-8 against 9.5e-8 here, states 5.3e-8 against
// 5.9e-8); jobs of more than 8 tokens have not been moved to it.
constexpr int kBlockTokens = 16;
constexpr int kQtStride = 20;  // row stride of Qt in floats: 16-byte rows whose vector stores do not collide
constexpr int kBlockCols = 32;  // columns of a CTA
constexpr size_t kChunkedSmemFloats = 2 * 4 * kBlockTokens * 64 + 64 * kQtStride + kBlockTokens * 64 + kBlockTokens * kBlockTokens + 64 +
                                      64 * kBlockCols + 4 * kBlockTokens * 64;
__global__ void __launch_bounds__(256) time_mix_v56_chunked_kernel(const WkvArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int S = 64, L = kBlockTokens, NC = kBlockCols;
    enum { IN_K = 0, IN_R = 1, IN_W = 2, IN_V = 3 };
    extern __shared__ __align__(16) float wkv_smem[];
    float(*sin)[4][L][S] = reinterpret_cast<float(*)[4][L][S]>(wkv_smem);              // [2]: staged k, r, w, v
    float(*Qt)[kQtStride] = reinterpret_cast<float(*)[kQtStride]>(wkv_smem + 2 * 4 * L * S);  // [S]: Qt[i][t] = r_t[i] Pe_t[i]
    float(*Kd)[S] = reinterpret_cast<float(*)[S]>(&Qt[S][0]);                            // [L]: Kd[s][i] = k_s[i] E_s[i]
    float(*At)[L] = reinterpret_cast<float(*)[L]>(&Kd[L][0]);                            // [L]: At[s][t] = A[t][s], 0 for s > t
    float* PL = &At[L][0];                                                               // [S]: the block's whole decay
    float(*S0)[NC] = reinterpret_cast<float(*)[NC]>(PL + S);                             // [S]: the state at the block's start
    float* red = &S0[S][0];  // [4][L][NC] partial outputs of the four key ranges; before that [L s][L t][16] partials of A
    __shared__ RunScratch run;
    const uint32_t tid = threadIdx.x;
    const uint32_t h = blockIdx.x / (S / NC), part = blockIdx.x % (S / NC), slot = blockIdx.y, C = a.S * a.H, c0 = h * S, v0 = part * NC;
    const uint32_t ri = tid / 16, cj = tid % 16;               // state tile: rows 4 ri .., columns 2 cj .. of the CTA's; keys 4 cj .. of A
    const uint32_t tg = tid / 64, tt = (tid % 64) / 8, oc = tid % 8;  // output tile: key range 16 tg .., tokens 2 tt .., columns 4 oc ..

    uint32_t start, count, carry;
    if (!find_run(a.cursors, a.wide, a.T, slot, &run, start, count, &carry)) return;
    if (carry != 0 && tid < NC)  // the carry row takes the layer input of the run's closing token (nothing here reads the row)
        static_cast<float*>(a.state.base)[a.state.index(c0 + v0 + tid, 0, slot)] = dload(a.x, a.dtype, (size_t)(carry - 1) * C + c0 + v0 + tid);

    float st[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
            st[r][cc] = static_cast<const float*>(a.state.base)[a.state.index(c0 + v0 + 2 * cj + cc, 1 + 4 * ri + r, slot)];
    float u4[4];  // time_first of the keys this thread takes in the A partials: 4 (tid % 16) ..
#pragma unroll
    for (int e = 0; e < 4; ++e) u4[e] = a.time_first[c0 + 4 * cj + e];

    // staging: thread (tensor = tid / 64, channel = tid % 64) takes the block's 16 tokens of its tensor and channel;
    // past the run's end k, r, v are 0 and w is 1 (such a token changes nothing).  The values stay as they were loaded until
    // store_chunk: anything done to one here would wait for it, and the loads would follow one another.
    uint32_t stage[L];
    const uint32_t tensor = tid / S, ch = tid % S;
    const void* src = tensor == IN_K ? a.k : tensor == IN_R ? a.r : tensor == IN_W ? (const void*)a.time_decay : a.v;
    const bool f16 = tensor != IN_W && a.dtype == WRK_F16;
    const size_t row = tensor == IN_W && !a.per_token_decay ? 0 : C, first = (size_t)start * row + c0 + ch;
    const uint32_t fill = tensor == IN_W ? 0x3f800000u : 0u;
    auto load_chunk = [&](uint32_t chunk) {
#pragma unroll
        for (int n = 0; n < L; ++n) stage[n] = fill;
        const uint32_t left = count - chunk * L;
        if (f16) {
            const unsigned short* p = static_cast<const unsigned short*>(src) + first + (size_t)chunk * L * row;
#pragma unroll
            for (int n = 0; n < L; ++n)
                if (n < left) stage[n] = p[n * row];
        } else {
            const uint32_t* p = static_cast<const uint32_t*>(src) + first + (size_t)chunk * L * row;
#pragma unroll
            for (int n = 0; n < L; ++n)
                if (n < left) stage[n] = p[n * row];
        }
    };
    auto store_chunk = [&](int buf) {
#pragma unroll
        for (int n = 0; n < L; ++n)
            sin[buf][tensor][n][ch] = f16 ? __half2float(__ushort_as_half((unsigned short)stage[n])) : __uint_as_float(stage[n]);
    };
    const uint32_t chunks = (count + L - 1) / L;
    load_chunk(0);
    store_chunk(0);
    __syncthreads();

    for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
        const int buf = chunk & 1;
        const bool more = chunk + 1 < chunks;
        if (more) load_chunk(chunk + 1);  // in flight while this block is computed
        const float(*sk)[S] = sin[buf][IN_K];
        const float(*sr)[S] = sin[buf][IN_R];
        const float(*sw)[S] = sin[buf][IN_W];
        const float(*sv)[S] = sin[buf][IN_V];

        // (1) the state tile to shared memory; the decay products; the partial sums of A
#pragma unroll
        for (int r = 0; r < 4; ++r) *reinterpret_cast<float2*>(&S0[4 * ri + r][2 * cj]) = make_float2(st[r][0], st[r][1]);
        {
            // thread (key i = tid % 64, quarter tq = tid / 64): Qt[i][4 tq ..], Kd[4 tq ..][i]; quarter 3 ends on the whole product
            const uint32_t i = tid % S, tq = tid / S;
            float pe = 1.0f;
#pragma unroll
            for (uint32_t t = 0; t < L - 4; ++t)
                if (t < 4 * tq) pe *= sw[t][i];
            float q[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                q[e] = sr[4 * tq + e][i] * pe;
                pe *= sw[4 * tq + e][i];
            }
            *reinterpret_cast<float4*>(&Qt[i][4 * tq]) = make_float4(q[0], q[1], q[2], q[3]);
            if (tq == 3) PL[i] = pe;
            float en = 1.0f;
#pragma unroll
            for (uint32_t s2 = L - 1; s2 > 3; --s2)
                if (s2 > 4 * tq + 3) en *= sw[s2][i];
#pragma unroll
            for (int e = 3; e >= 0; --e) {
                Kd[4 * tq + e][i] = sk[4 * tq + e][i] * en;
                en *= sw[4 * tq + e][i];
            }
        }
        {
            // thread (s = tid / 16, keys 4 cj ..): its share of A[t][s] for t = s .. L - 1, into red[s][t][cj]
            const uint32_t s2 = tid / 16;
            const float4 kq = *reinterpret_cast<const float4*>(&sk[s2][4 * cj]);
            const float kk[4] = {kq.x, kq.y, kq.z, kq.w};
            float d[4] = {1.0f, 1.0f, 1.0f, 1.0f};
            for (uint32_t t = 0; t < s2; ++t) red[(s2 * L + t) * 16 + cj] = 0.0f;
            {
                const float4 rq = *reinterpret_cast<const float4*>(&sr[s2][4 * cj]);
                red[(s2 * L + s2) * 16 + cj] = (rq.x * kk[0] * u4[0] + rq.y * kk[1] * u4[1]) + (rq.z * kk[2] * u4[2] + rq.w * kk[3] * u4[3]);
            }
            // (not unrolled by hand: a peeled first step, d = 1, would let the compiler fuse other products)
            for (uint32_t t = s2 + 1; t < L; ++t) {
                const float4 rq = *reinterpret_cast<const float4*>(&sr[t][4 * cj]);
                const float4 wq = *reinterpret_cast<const float4*>(&sw[t][4 * cj]);
                red[(s2 * L + t) * 16 + cj] = (rq.x * kk[0] * d[0] + rq.y * kk[1] * d[1]) + (rq.z * kk[2] * d[2] + rq.w * kk[3] * d[3]);
                d[0] *= wq.x, d[1] *= wq.y, d[2] *= wq.z, d[3] *= wq.w;
            }
        }
        __syncthreads();
        // (2) A[t][s] summed over the 16 key groups: thread (s, t) = (tid / 16, tid % 16)
        {
            const float4* p4 = reinterpret_cast<const float4*>(red + (size_t)tid * 16);
            const float4 p0 = p4[0], p1 = p4[1], p2 = p4[2], p3 = p4[3];
            At[tid / 16][tid % 16] = ((p0.x + p0.y) + (p0.z + p0.w)) + ((p1.x + p1.y) + (p1.z + p1.w)) +
                                     (((p2.x + p2.y) + (p2.z + p2.w)) + ((p3.x + p3.y) + (p3.z + p3.w)));
        }
        __syncthreads();
        // (3) the outputs of tokens 2 tt .. and columns 4 oc .., summed over keys 16 tg .. (the state's share) and over the
        // block's tokens 4 tg .. (their own share); then the new state tile
        {
            float acc[2][4];
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) acc[e][cc] = 0.0f;
#pragma unroll 8
            for (uint32_t i = 16 * tg; i < 16 * tg + 16; ++i) {
                const float2 q2 = *reinterpret_cast<const float2*>(&Qt[i][2 * tt]);
                const float4 s4 = *reinterpret_cast<const float4*>(&S0[i][4 * oc]);
                const float qv[2] = {q2.x, q2.y}, sv4[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) acc[e][cc] = fmaf(qv[e], sv4[cc], acc[e][cc]);
            }
#pragma unroll
            for (uint32_t s2 = 4 * tg; s2 < 4 * tg + 4; ++s2) {
                const float2 a2 = *reinterpret_cast<const float2*>(&At[s2][2 * tt]);
                const float4 v4 = *reinterpret_cast<const float4*>(&sv[s2][v0 + 4 * oc]);
                const float av[2] = {a2.x, a2.y}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) acc[e][cc] = fmaf(av[e], vv[cc], acc[e][cc]);
            }
            // red is free again: every thread has passed the barrier that follows its last read in (2)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                *reinterpret_cast<float4*>(&red[((size_t)tg * L + 2 * tt + e) * NC + 4 * oc]) = make_float4(acc[e][0], acc[e][1], acc[e][2], acc[e][3]);
        }
        {
            const float4 pl = *reinterpret_cast<const float4*>(&PL[4 * ri]);
            const float plv[4] = {pl.x, pl.y, pl.z, pl.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) st[r][cc] *= plv[r];
#pragma unroll 8
            for (uint32_t s2 = 0; s2 < L; ++s2) {
                const float4 k4 = *reinterpret_cast<const float4*>(&Kd[s2][4 * ri]);
                const float2 v2 = *reinterpret_cast<const float2*>(&sv[s2][v0 + 2 * cj]);
                const float kv[4] = {k4.x, k4.y, k4.z, k4.w}, vv[2] = {v2.x, v2.y};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) st[r][cc] = fmaf(kv[r], vv[cc], st[r][cc]);
            }
        }
        __syncthreads();
        // (4) token t = tid / 16, columns 2 cj ..: the four key ranges' partial outputs
        {
            const uint32_t t = tid / 16, m = chunk * L + t;
            if (m < count) {
                float2 y = *reinterpret_cast<const float2*>(&red[((size_t)0 * L + t) * NC + 2 * cj]);
#pragma unroll
                for (int g = 1; g < 4; ++g) {
                    const float2 p = *reinterpret_cast<const float2*>(&red[((size_t)g * L + t) * NC + 2 * cj]);
                    y.x += p.x, y.y += p.y;
                }
                const size_t ti = (size_t)(start + m) * C + c0 + v0 + 2 * cj;
                dstore(a.x, a.dtype, ti, y.x);
                dstore(a.x, a.dtype, ti + 1, y.y);
            }
        }
        if (more) store_chunk(buf ^ 1);  // last read during the previous block, before its closing barrier
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
            static_cast<float*>(a.state.base)[a.state.index(c0 + v0 + 2 * cj + cc, 1 + 4 * ri + r, slot)] = st[r][cc];
}

// v7: a CTA takes NC columns of a head's state, as above.  NC S / RPT threads compute: a thread keeps RPT rows of one column
// (quads of rows S / RPT quads apart, so that the row groups' shared-memory reads meet no bank twice), the S / RPT row
// groups of a column are neighbouring lanes; `sa` is summed over them in log2(S / RPT) shuffles per token, the outputs of
// four tokens together.  Four more warps fetch the tokens' rows a chunk ahead, apply the per-token transforms
// (w -> exp(-0.606531 sigmoid(w)), -kk, kk a) and hand them over through shared memory, one barrier per chunk.
// Measured at 64 heads of 64, one sequence of 256 tokens: 62 us (0.23 us per further token); a thread per whole column, on
// 64 SMs, took 113 us; eight rows per thread and twice the warps 66 us.
constexpr int kV7Loaders = 128;
// tokens of a chunk: two chunks fit 47 KB of shared memory
template <int S, int NC>
constexpr int kV7Chunk = 128 * (5 * S + NC) <= 47 * 1024 ? 16 : 64 * (5 * S + NC) <= 47 * 1024 ? 8 : 4;
template <int S, int NC, int RPT>
__global__ void __launch_bounds__(NC * (S / RPT) + kV7Loaders) time_mix_v7_kernel(const WkvArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int RG = S / RPT, NT = NC * RG, TC = kV7Chunk<S, NC>, QUADS = S / 4, QT = (TC * QUADS + kV7Loaders - 1) / kV7Loaders;
    enum { IN_R = 0, IN_W = 1, IN_K = 2, IN_A = 3, IN_B = 4 };
    __shared__ __align__(16) float sin[2][5][TC][S], sv[2][TC][NC];
    __shared__ RunScratch run;
    const uint32_t tid = threadIdx.x, rg = tid % RG, col = tid / RG;
    const uint32_t h = blockIdx.x / (S / NC), part = blockIdx.x % (S / NC), slot = blockIdx.y, C = a.S * a.H, c0 = h * S, v0 = c0 + part * NC;
    const size_t plane = (size_t)a.T * C;

    uint32_t start, count, carry;
    if (!find_run(a.cursors, a.wide, a.T, slot, &run, start, count, &carry)) return;
    // the carry row takes the layer input of the run's closing token: written now (nothing here reads the row), before
    // the token's input is overwritten with its output
    if (carry != 0 && tid < NC)
        static_cast<float*>(a.state.base)[a.state.index(v0 + tid, 0, slot)] = dload(a.x, a.dtype, (size_t)(carry - 1) * C + v0 + tid);

    const uint32_t chunks = (count + TC - 1) / TC;
    if (tid >= NT) {
        const uint32_t lid = tid - NT;
        auto decay = [](float w) { return expf(-0.606531f * (1.0f / (1.0f + expf(-w)))); };
        // (token, four channels) pairs lid, lid + kV7Loaders, ... of the chunk; zero past the run's end
        auto stage = [&](uint32_t chunk) {
            float4 gr[QT], gw[QT], gk[QT], ga[QT], gkk[QT], gv[QT];
#pragma unroll
            for (int q = 0; q < QT; ++q) {
                const uint32_t idx = lid + q * kV7Loaders, m = chunk * TC + idx / QUADS, c = 4 * (idx % QUADS);
                gr[q] = gw[q] = gk[q] = ga[q] = gkk[q] = gv[q] = splat4(0.f);
                if (idx < TC * QUADS && m < count) {
                    const size_t ti = (size_t)(start + m) * C;
                    gr[q] = load_quad(a.r, a.dtype, ti + c0 + c);
                    gw[q] = load_quad(a.w, a.dtype, ti + c0 + c);
                    gk[q] = load_quad(a.n, a.dtype, ti + c0 + c);
                    ga[q] = load_quad(a.n, a.dtype, ti + c0 + c + 2 * plane);
                    gkk[q] = load_quad(a.n, a.dtype, ti + c0 + c + 3 * plane);
                    if (c < NC) gv[q] = load_quad(a.n, a.dtype, ti + v0 + c + plane);
                }
            }
            const int buf = chunk & 1;
#pragma unroll
            for (int q = 0; q < QT; ++q) {
                const uint32_t idx = lid + q * kV7Loaders, n = idx / QUADS, c = 4 * (idx % QUADS);
                if (idx >= TC * QUADS) break;
                *reinterpret_cast<float4*>(&sin[buf][IN_R][n][c]) = gr[q];
                *reinterpret_cast<float4*>(&sin[buf][IN_W][n][c]) = make_float4(decay(gw[q].x), decay(gw[q].y), decay(gw[q].z), decay(gw[q].w));
                *reinterpret_cast<float4*>(&sin[buf][IN_K][n][c]) = gk[q];
                *reinterpret_cast<float4*>(&sin[buf][IN_A][n][c]) = make_float4(-gkk[q].x, -gkk[q].y, -gkk[q].z, -gkk[q].w);
                *reinterpret_cast<float4*>(&sin[buf][IN_B][n][c]) =
                    make_float4(gkk[q].x * ga[q].x, gkk[q].y * ga[q].y, gkk[q].z * ga[q].z, gkk[q].w * ga[q].w);
                if (c < NC) *reinterpret_cast<float4*>(&sv[buf][n][c]) = gv[q];
            }
        };
        stage(0);
        __syncthreads();
#pragma unroll 1
        for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
            if (chunk + 1 < chunks) stage(chunk + 1);  // that buffer was last read two chunks ago, before that chunk's closing barrier
            __syncthreads();
        }
        return;
    }

    float2 st[RPT / 2];
    auto row = [&](uint32_t i) { return 1 + 4 * ((i / 2) * RG + rg) + 2 * (i % 2); };  // state row of st[i].x; st[i].y is the next
#pragma unroll
    for (int i = 0; i < RPT / 2; ++i)
        st[i] = make_float2(static_cast<const float*>(a.state.base)[a.state.index(v0 + col, row(i), slot)],
                            static_cast<const float*>(a.state.base)[a.state.index(v0 + col, row(i) + 1, slot)]);
    auto token = [&](int buf, uint32_t n) {
        const float4* r4 = reinterpret_cast<const float4*>(sin[buf][IN_R][n]) + rg;
        const float4* w4 = reinterpret_cast<const float4*>(sin[buf][IN_W][n]) + rg;
        const float4* k4 = reinterpret_cast<const float4*>(sin[buf][IN_K][n]) + rg;
        const float4* a4 = reinterpret_cast<const float4*>(sin[buf][IN_A][n]) + rg;
        const float4* b4 = reinterpret_cast<const float4*>(sin[buf][IN_B][n]) + rg;
        float2 z0 = make_float2(0.f, 0.f), z1 = z0;
#pragma unroll
        for (int i = 0; i < RPT / 4; ++i) {
            const float4 av = a4[i * RG];
            z0 = __ffma2_rn(st[2 * i], lo2(av), z0);
            z1 = __ffma2_rn(st[2 * i + 1], hi2(av), z1);
        }
        float sa = (z0.x + z0.y) + (z1.x + z1.y);
#pragma unroll
        for (int mask = 1; mask < RG; mask *= 2) sa += __shfl_xor_sync(0xffffffffu, sa, mask);
        const float vj = sv[buf][n][col];
        const float2 v2 = make_float2(vj, vj), sa2 = make_float2(sa, sa);
        float2 y0 = make_float2(0.f, 0.f), y1 = y0;
#pragma unroll
        for (int i = 0; i < RPT / 4; ++i) {
            const float4 wv = w4[i * RG], kv = k4[i * RG], bv = b4[i * RG], rv = r4[i * RG];
            st[2 * i] = __ffma2_rn(sa2, lo2(bv), __ffma2_rn(lo2(kv), v2, __fmul2_rn(st[2 * i], lo2(wv))));
            st[2 * i + 1] = __ffma2_rn(sa2, hi2(bv), __ffma2_rn(hi2(kv), v2, __fmul2_rn(st[2 * i + 1], hi2(wv))));
            y0 = __ffma2_rn(lo2(rv), st[2 * i], y0);
            y1 = __ffma2_rn(hi2(rv), st[2 * i + 1], y1);
        }
        return (y0.x + y0.y) + (y1.x + y1.y);
    };
    __syncthreads();
#pragma unroll 1
    for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
        const int buf = chunk & 1;
        const uint32_t len = min((uint32_t)TC, count - chunk * TC), t0 = start + chunk * TC;
#pragma unroll 1
        for (uint32_t n0 = 0; n0 < len; n0 += 4) {
            float y[4];
#pragma unroll
            for (uint32_t n = 0; n < 4; ++n) {
                y[n] = 0.f;
                if (n0 + n < len) y[n] = token(buf, n0 + n);  // the same for every thread
            }
            sum_scatter<4, RG>(y, rg);
            constexpr uint32_t OUT = RG <= 4 ? 4 / RG : 1, COPIES = RG <= 4 ? 1 : RG / 4;
#pragma unroll
            for (uint32_t e = 0; e < OUT; ++e) {
                const uint32_t n = rg * 4 / RG + e;
                if (rg % COPIES == 0 && n0 + n < len) dstore(a.x, a.dtype, (size_t)(t0 + n0 + n) * C + v0 + col, y[e]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < RPT / 2; ++i) {
        static_cast<float*>(a.state.base)[a.state.index(v0 + col, row(i), slot)] = st[i].x;
        static_cast<float*>(a.state.base)[a.state.index(v0 + col, row(i) + 1, slot)] = st[i].y;
    }
}

// v7, runs of a few tokens (batched decode: many sequences, a token or two each): S threads per (head, batch slot),
// thread j with column j of the state, a token's shared vectors through double-buffered shared memory.  Such a job
// streams the states (S x S floats per head and sequence, in and out) and little else; the small CTA keeps six of
// them on an SM where the staged kernel above fits one.
template <int S>
__global__ void __launch_bounds__(S) time_mix_v7_short_kernel(const WkvArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float sr[2][S], sw[2][S], sk[2][S], sa[2][S], sb[2][S];
    __shared__ RunScratch run;
    const uint32_t h = blockIdx.x, slot = blockIdx.y, j = threadIdx.x;
    const uint32_t C = a.S * a.H, c = h * S + j;
    const size_t plane = (size_t)a.T * C;

    uint32_t start, count;
    if (!find_run(a.cursors, a.wide, a.T, slot, &run, start, count)) return;

    float st[S];
#pragma unroll
    for (int i = 0; i < S; ++i) st[i] = static_cast<const float*>(a.state.base)[a.state.index(c, 1 + i, slot)];

    auto decay = [](float w) { return expf(-0.606531f * (1.0f / (1.0f + expf(-w)))); };
    {
        const size_t ti = (size_t)start * C + c;
        sr[0][j] = dload(a.r, a.dtype, ti);
        sw[0][j] = decay(dload(a.w, a.dtype, ti));
        sk[0][j] = dload(a.n, a.dtype, ti);
        const float av = dload(a.n, a.dtype, ti + 2 * plane), kk = dload(a.n, a.dtype, ti + 3 * plane);
        sa[0][j] = -kk;
        sb[0][j] = kk * av;
    }
    __syncthreads();

    for (uint32_t n = 0; n < count; ++n) {
        const uint32_t t = start + n;
        const int cur = n & 1, nxt = cur ^ 1;
        const size_t ti = (size_t)t * C + c;
        const bool more = n + 1 < count;
        float nr = 0.f, nw = 0.f, nk = 0.f, na = 0.f, nkk = 0.f;
        if (more) {
            nr = dload(a.r, a.dtype, ti + C);
            nw = dload(a.w, a.dtype, ti + C);
            nk = dload(a.n, a.dtype, ti + C);
            na = dload(a.n, a.dtype, ti + C + 2 * plane);
            nkk = dload(a.n, a.dtype, ti + C + 3 * plane);
        }
        const float vj = dload(a.n, a.dtype, ti + plane);
        const float xin = dload(a.x, a.dtype, ti);
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int i = 0; i < S; i += 4) {
            s0 = fmaf(st[i], sa[cur][i], s0);
            s1 = fmaf(st[i + 1], sa[cur][i + 1], s1);
            s2 = fmaf(st[i + 2], sa[cur][i + 2], s2);
            s3 = fmaf(st[i + 3], sa[cur][i + 3], s3);
        }
        const float sav = (s0 + s1) + (s2 + s3);
        float y0 = 0.f, y1 = 0.f, y2 = 0.f, y3 = 0.f;
#pragma unroll
        for (int i = 0; i < S; i += 4) {
            st[i] = st[i] * sw[cur][i] + sk[cur][i] * vj + sav * sb[cur][i];
            y0 = fmaf(sr[cur][i], st[i], y0);
            st[i + 1] = st[i + 1] * sw[cur][i + 1] + sk[cur][i + 1] * vj + sav * sb[cur][i + 1];
            y1 = fmaf(sr[cur][i + 1], st[i + 1], y1);
            st[i + 2] = st[i + 2] * sw[cur][i + 2] + sk[cur][i + 2] * vj + sav * sb[cur][i + 2];
            y2 = fmaf(sr[cur][i + 2], st[i + 2], y2);
            st[i + 3] = st[i + 3] * sw[cur][i + 3] + sk[cur][i + 3] * vj + sav * sb[cur][i + 3];
            y3 = fmaf(sr[cur][i + 3], st[i + 3], y3);
        }
        const CursorD cu = cursor_at(a.cursors, a.wide, t);
        if (t - cu.token + 1u == cu.len)
            static_cast<float*>(a.state.base)[a.state.index(c, 0, slot)] = xin;
        dstore(a.x, a.dtype, ti, (y0 + y1) + (y2 + y3));
        if (more) {
            sr[nxt][j] = nr;
            sw[nxt][j] = decay(nw);
            sk[nxt][j] = nk;
            sa[nxt][j] = -nkk;
            sb[nxt][j] = nkk * na;
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < S; ++i) static_cast<float*>(a.state.base)[a.state.index(c, 1 + i, slot)] = st[i];
}

// x_j += (sum_i u_i k_i r_i) * v_j per (token, head): one warp per (token, head).
__global__ void time_first_v7_kernel(const __half* u, int dtype, const void* r, const void* n, void* x, uint32_t S,
                                     uint32_t H, uint32_t T) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= T * H) return;
    const uint32_t t = warp / H, h = warp % H;
    const uint32_t C = S * H;
    const size_t base = (size_t)t * C + h * S, plane = (size_t)T * C;
    float s = 0.f;
    for (uint32_t i = lane; i < S; i += 32)
        s += __half2float(u[h * S + i]) * dload(n, dtype, base + i) * dload(r, dtype, base + i);
    s = warp_sum(s);
    for (uint32_t i = lane; i < S; i += 32)
        dstore(x, dtype, base + i, dload(x, dtype, base + i) + s * dload(n, dtype, base + i + plane));
}

}  // namespace

// A job's kernels start early, on the SMs that the kernels before them leave free: CTAs that then compute for a long time
// sit several to an SM.  With more than 64 tokens the recurrence waits for the kernel before it to end (256 tokens of one
// sequence among four slots, 40 heads: 60 us when started early, against 35 alone; a launch that waits costs about 2 us).
static bool wkv_early(const WkvArgs& a) { return a.T <= 64; }

// A head's columns are shared out among CTAs unless the outputs overwrite an input that every CTA of the head reads.
cudaError_t time_mix_v56(const WkvArgs& a, cudaStream_t stream) {
    if (a.T == 0 || a.B == 0) return cudaSuccess;
    const bool whole = a.x == a.k || a.x == a.r || a.x == a.time_decay, early = wkv_early(a);
    if (a.S == 32) launch_early(early, time_mix_v56_kernel<32, 32>, dim3(a.H, a.B), dim3(64), 0, stream, a);
    else if (a.S == 64 && whole) launch_early(early, time_mix_v56_kernel<64, 64>, dim3(a.H, a.B), dim3(256), 0, stream, a);
    else if (a.S == 64) launch_early(early, time_mix_v56_kernel<64, 32>, dim3(2 * a.H, a.B), dim3(128), 0, stream, a);
    else if (a.S == 128 && whole) launch_early(early, time_mix_v56_kernel<128, 128>, dim3(a.H, a.B), dim3(1024), 0, stream, a);
    else if (a.S == 128) launch_early(early, time_mix_v56_kernel<128, 32>, dim3(4 * a.H, a.B), dim3(256), 0, stream, a);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// The block form of time_mix_v56: heads of 64 channels whose outputs overwrite no input that both CTAs of a head read.
bool time_mix_v56_chunked_supported(const WkvArgs& a) { return a.S == 64 && a.x != a.k && a.x != a.r && a.x != a.time_decay; }

cudaError_t time_mix_v56_chunked(const WkvArgs& a, cudaStream_t stream) {
    if (a.T == 0 || a.B == 0) return cudaSuccess;
    if (!time_mix_v56_chunked_supported(a)) return cudaErrorInvalidValue;
    static SmemOptIn opt_in;
    const size_t smem = kChunkedSmemFloats * sizeof(float);
    if (cudaError_t e = opt_in.ensure(time_mix_v56_chunked_kernel, (int)smem); e != cudaSuccess) return e;
    launch_early(wkv_early(a), time_mix_v56_chunked_kernel, dim3(a.S / kBlockCols * a.H, a.B), dim3(256), smem, stream, a);
    return cudaGetLastError();
}

cudaError_t time_mix_v7(const WkvArgs& a, cudaStream_t stream) {
    if (a.T == 0 || a.B == 0) return cudaSuccess;
    dim3 grid(a.H, a.B);
    if (a.T <= 4 * a.B) {  // at most four tokens per sequence on average
        switch (a.S) {
            case 32: launch(time_mix_v7_short_kernel<32>, grid, dim3(32), 0, stream, a); break;
            case 64: launch(time_mix_v7_short_kernel<64>, grid, dim3(64), 0, stream, a); break;
            case 128: launch(time_mix_v7_short_kernel<128>, grid, dim3(128), 0, stream, a); break;
            default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
    const bool whole = a.x == a.r || a.x == a.w || a.x == a.n, early = wkv_early(a);  // as in time_mix_v56
    constexpr int L = kV7Loaders;
    if (a.S == 32) launch_early(early, time_mix_v7_kernel<32, 32, 16>, grid, dim3(64 + L), 0, stream, a);
    else if (a.S == 64 && whole) launch_early(early, time_mix_v7_kernel<64, 64, 16>, grid, dim3(256 + L), 0, stream, a);
    else if (a.S == 64) launch_early(early, time_mix_v7_kernel<64, 32, 16>, dim3(2 * a.H, a.B), dim3(128 + L), 0, stream, a);
    else if (a.S == 128 && whole) launch_early(early, time_mix_v7_kernel<128, 128, 32>, grid, dim3(512 + L), 0, stream, a);
    else if (a.S == 128) launch_early(early, time_mix_v7_kernel<128, 32, 16>, dim3(4 * a.H, a.B), dim3(256 + L), 0, stream, a);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// time_mix_v4.wgsl: per channel c and token t (batch from the cursor), with (aa, bb, pp) = state rows 1..3:
//   x_t = sigmoid(r_t) * (e1 aa + e2 v_t) / (e1 bb + e2),   e1 = exp(pp - q), e2 = exp(u + k_t - q), q = max(pp, u + k_t)
//   (aa, bb, pp) <- (e1' aa + e2' v_t, e1' bb + e2', q'),      e1' = exp(w + pp - q'), e2' = exp(k_t - q'), q' = max(w + pp, k_t)
// and state row 0 <- the input x of the sequence's last token in the job.  One thread per channel walks the tokens in
// order and keeps (aa, bb, pp) in registers while consecutive tokens belong to one batch slot.
__global__ void time_mix_v4_kernel(const uint32_t* cursors, int wide, const float* time_decay, const float* time_first,
                                   DView state, int dtype, const void* k, const void* v, const void* r, void* x,
                                   uint32_t C, uint32_t T) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const float u = time_first[c], w = time_decay[c];
    float* st = static_cast<float*>(state.base);
    uint32_t held = 0xffffffffu;  // batch slot whose recurrence is in registers
    float aa = 0.f, bb = 0.f, pp = 0.f;
    for (uint32_t t = 0; t < T; ++t) {
        const CursorD cu = cursor_at(cursors, wide, t);
        if (cu.batch != held) {
            if (held != 0xffffffffu) {
                st[state.index(c, 1, held)] = aa;
                st[state.index(c, 2, held)] = bb;
                st[state.index(c, 3, held)] = pp;
            }
            held = cu.batch;
            aa = st[state.index(c, 1, held)];
            bb = st[state.index(c, 2, held)];
            pp = st[state.index(c, 3, held)];
        }
        const size_t ti = (size_t)t * C + c;
        // the token-shift carry: read before this token's slot of x is overwritten (the last token's slot is >= t)
        const uint32_t last = cu.token + cu.len - 1u;
        if ((t == last || t == cu.token) && last >= t && last < T)
            st[state.index(c, 0, held)] = dload(x, dtype, (size_t)last * C + c);
        const float kk = dload(k, dtype, ti), vv = dload(v, dtype, ti);
        const float rr = 1.0f / (1.0f + expf(-dload(r, dtype, ti)));
        float ww = u + kk;
        float q = fmaxf(pp, ww);
        float e1 = expf(pp - q), e2 = expf(ww - q);
        dstore(x, dtype, ti, rr * (e1 * aa + e2 * vv) / (e1 * bb + e2));
        ww = w + pp;
        q = fmaxf(ww, kk);
        e1 = expf(ww - q);
        e2 = expf(kk - q);
        aa = e1 * aa + e2 * vv;
        bb = e1 * bb + e2;
        pp = q;
    }
    if (held != 0xffffffffu) {
        st[state.index(c, 1, held)] = aa;
        st[state.index(c, 2, held)] = bb;
        st[state.index(c, 3, held)] = pp;
    }
}

cudaError_t time_mix_v4(const uint32_t* cursors, int wide, const float* time_decay, const float* time_first, DView state,
                        int dtype, const void* k, const void* v, const void* r, void* x, uint32_t C, uint32_t T,
                        cudaStream_t stream) {
    if (T == 0 || C == 0) return cudaSuccess;
    launch(time_mix_v4_kernel, dim3((C + 127) / 128), dim3(128), 0, stream, cursors, wide, time_decay, time_first, state, dtype, k, v, r, x, C, T);
    return cudaGetLastError();
}

cudaError_t time_first_v7(const __half* u, int dtype, const void* r, const void* n, void* x, uint32_t S, uint32_t H,
                          uint32_t T, cudaStream_t stream) {
    if (T == 0) return cudaSuccess;
    const uint32_t warps = T * H;
    const uint32_t blocks = (warps * 32 + 255) / 256;
    launch(time_first_v7_kernel, dim3(blocks), dim3(256), 0, stream, u, dtype, r, n, x, S, H, T);
    return cudaGetLastError();
}

}  // namespace k
}  // namespace wrk
