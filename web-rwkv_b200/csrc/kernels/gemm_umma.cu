// Tensor-memory GEMM for the prefill / batched path (matmul_mat_fp16 / int8 / nf4 with 16 or more tokens):
// out[n][m] = act(sum_k W[m][k] * x[n][k]).
//
// One CTA owns a 128-row slice of W and up to 256 tokens and walks K in steps of 64.  Warp roles:
//   * warp 9 (one thread) streams the packed weight tiles with TMA: 128 rows x 128 (Int8) or 64 (NF4) bytes per pair of
//     steps into a swizzled ring of raw stages; fp16 weights go straight into the A operand stage;
//   * warp 10 (one thread) streams the fp16 activations, [steps][tokens][64] per copy, into the B operand stages (rows
//     past the last token are zero-filled by the TMA unit);
//   * warps 0-7 dequantize as two groups of four warps on alternate pairs of steps: a thread owns a row of the tile, turns
//     its 64 weights of a step into fp16 (f32 math, one rounding) and stores them in TENSOR MEMORY, 32 columns per step:
//     the A operand of the MMA, row m in lane m;
//   * warp 8 (one thread) issues tcgen05.mma.cta_group::1.kind::f16 (M = 128, N = token tile, K = 16, four per step) into
//     an accumulator of 128 lanes x N fp32 columns and releases the stages with tcgen05.commit;
//   * after the last step warps 0-7 bring the accumulator to shared memory (the operand stages are free by then), and all
//     warps write it out, four rows of a token per thread.
// A launch takes up to four matrices of one format, K and token count (UmmaGroup): their row tiles share grid.x, so
// key / value / receptance / gate of a layer fill the SMs together and none has to split K.
// Where the output tiles alone leave SMs idle, the CTAs of a thread-block cluster (up to 8, along grid.z) split the
// K range of one tile; after a cluster barrier CTA r finishes its share of the columns, adding its peers' partial tiles
// through distributed shared memory.
// Weights enter the MMA as fp16(fma(q, (max - min) / 255, min)) resp. fp16(table[nib] * absmax), computed in
// f32 and rounded once; the accumulation is fp32.  Every wait on an mbarrier is bounded: on a timeout the
// kernel records WRK_ERR_TIMEOUT in the context's status word, stops waiting and copying, lets the copies and MMAs in flight
// end (with a limit again) and still frees its TMEM.  A wait whose end
// depends on the activations comes after griddepcontrol.wait: the limit does not count the kernels in front.
//
// What bounds it: at 256 tokens a step is 512 cycles of MMA; it takes about 850, most of it shared-memory and L2 traffic of the
// activation tile (32 KB per step and CTA).  At 64 tokens and below the dequantizers' instructions (about 250 cycles per
// step) and the HBM stream of the weights are of one size, and a launch has about 5 us of fixed work.  An operand A that
// went through shared memory cost 32 KB of its traffic per step and a proxy fence; what cost more was the issuing
// threads: per step, divisions by ring sizes, parameters read again from memory, barrier answers waited for one after
// the other and `lane == 0` branches around tensor-core instructions took 1100 cycles.  Measured with and without all of
// these (us; Int8 unless noted): four 4096 x 4096 at 256 tokens 57 -> 35, 4096 x 14336 at 256 tokens 54 -> 34, 16384 x 4096
// at 64 tokens 44 -> 23, 768 x 768 at 32 tokens 12 -> 5; NF4 four 2560 x 2560 at 256 tokens 47 -> 23; fp16 65536 x 2048 at
// 16 tokens 71 -> 48 (5.6 TB/s), 14336 x 4096 at 1024 tokens 158 -> 139.
#include <cuda.h>

#include "device.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace wrk {
namespace k {

namespace {

constexpr int BM = 128;             // weight rows per CTA (UMMA M)
constexpr int BK = 64;              // K per step: one 128-byte swizzle atom of fp16 activations
constexpr int kDequantWarps = 8;
constexpr int kMmaWarp = 8, kWeightTmaWarp = 9;  // warp 10 streams the activations
constexpr int kUmmaThreads = 11 * 32;
constexpr int kMaxStages = 8;       // operand stages
constexpr int kMaxRaw = 8;          // raw weight stages
constexpr uint32_t kScaleSlots = 8, kScaleAhead = 6;
constexpr uint32_t SCALE_BYTES = 2 * kScaleSlots * BM * 4;  // two groups of dequantizing warps
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr uint32_t kDrainLimit = 1u << 16;
constexpr uint32_t kSplitSmem = 114 * 1024;  // half of the 228 KB of an SM; 1 KB more per CTA is the system's
constexpr uint32_t A_STEP_BYTES = BM * BK * 2;  // fp16 weights: 16 KB of shared memory per step
constexpr uint32_t A_STEP_COLS = BK / 2;        // quantized weights: 32 TMEM columns of fp16 pairs per step

// Up to kMaxGroup problems of one weight format, K, token count and tiling in one launch: the row tiles of problem i
// are CTAs tile_start[i] .. tile_start[i + 1] - 1 along grid.x.  Matrices that read different activations at the same
// point of a layer (key / value / receptance / gate) fill the SMs together, where each alone would have to split K
// and pay for the exchange of partial tiles.
constexpr int kMaxGroup = 4;
struct UmmaProblem {
    const __half* scale;
    const float* table;
    uint32_t M;
    int act;
    DView out;
};
struct alignas(64) UmmaGroup {
    CUtensorMap map_w[kMaxGroup], map_x[kMaxGroup];
    UmmaProblem p[kMaxGroup];
    uint32_t tile_start[kMaxGroup + 1];
    uint32_t count;
    uint32_t K, N;
    uint32_t n_tile;     // tokens per CTA: multiple of 16, <= 256
    uint32_t acc_cols;   // accumulator columns: n_tile rounded up to 32
    uint32_t tmem_cols;  // power of two: the accumulator and, for quantized weights, the A stages
    uint32_t bu;         // steps per stage of the activation operand (and of fp16 weights): 1 or 2
    uint32_t a_stages;   // quantized weights: A stages in tensor memory, a pair of steps each
    uint32_t b_stages;   // activation stages (fp16 weights: of both operands)
    uint32_t raw;        // raw weight stages (quantized kinds), a pair of steps each
    uint32_t splits;     // CTAs along K per output tile (grid.z = the cluster's size)
    int32_t* status;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// A position in a ring of stages: the stage and the parity of its current use.  Counted, not divided: a division by the
// number of stages in every step cost the issuing thread more than the tensor core's work.
struct Ring {
    uint32_t stage = 0, phase = 0;
    __device__ __forceinline__ void next(uint32_t stages) {
        if (++stage == stages) stage = 0, phase ^= 1;
    }
    __device__ __forceinline__ void skip(uint32_t n, uint32_t stages) {  // n <= stages
        stage += n;
        if (stage >= stages) stage -= stages, phase ^= 1;
    }
};

// True in one lane of the (converged) warp.  The compiler knows the branch is taken by one thread, which keeps the operands
// of the tensor-core instructions in uniform registers; behind `lane == 0` each tcgen05.mma cost its thread 0.1 us.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(pred));
    return pred != 0;
}
// Tiled TMA load of the box at (x, y (, z)) into this CTA's shared memory at dst, completing on bar.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void cp_async4z(void* dst, const void* src, bool valid) {
    const uint32_t n = valid ? 4u : 0u;  // src-size 0: zero-filled, nothing is read
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}
// Whether the phase with the given parity has completed, now (test) or within a short time (try, which may suspend the
// thread).  The answer takes some 60 cycles: a thread that tests the next stage before it works on this one does not wait
// for it.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for it; gives up (false) after kSpinLimit polls (or at once when another wait of this CTA has already given up) and
// reports it.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    if (status != nullptr) atomicExch(status, (int32_t)WRK_ERR_TIMEOUT);
    return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle (start address, LBO = 1, SBO = 1024 bytes, version 1, SWIZZLE_128B).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// Instruction descriptor: fp16 x fp16 -> fp32, both operands K-major, M x N.
__device__ __forceinline__ uint32_t f16_idesc(uint32_t m, uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with the A operand in tensor memory: row m in lane m, two consecutive K elements per 32-bit column.
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t v[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// Four activations, out of line: the copy-out loop stays short.
__device__ __noinline__ float4 activate4(int act, float4 v) {
    return make_float4(activate_f(act, v.x), activate_f(act, v.y), activate_f(act, v.z), activate_f(act, v.w));
}
// 32 columns of this warp's 32 lanes; waits until the store has been performed.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t v[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
        "tcgen05.wait::st.sync.aligned;\n" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
        "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// Thread-block cluster: hardware barrier over all threads of all CTAs of the cluster, and 16-byte loads from
// a peer CTA's shared memory.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ float4 ld_peer_smem(uint32_t local_addr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local_addr), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(remote)
                 : "memory");
    return v;
}

__device__ __forceinline__ uint32_t pack_half2(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// 16 Int8 weights of one row (16 raw bytes), slope and minimum of their block -> 8 fp16 pairs.  f32 arithmetic, one
// rounding to fp16 per weight: the errors of a row are independent, none is shared by a whole block.
__device__ __forceinline__ void dequant_int8(uint4 q, float sc, float mn, uint32_t* h) {
    const uint32_t words[4] = {q.x, q.y, q.z, q.w};
    const float2 sc2 = make_float2(sc, sc), mn2 = make_float2(mn, mn), bias2 = make_float2(-8388608.0f, -8388608.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // byte b -> float 8388608 + b (0x4B000000 | b), minus 8388608: b exactly; two weights per instruction from
        // there on (add.f32x2, fma.rn.f32x2: the same roundings as the scalar forms)
        const float2 f01 = make_float2(__uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7650)),
                                       __uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7651)));
        const float2 f23 = make_float2(__uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7652)),
                                       __uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7653)));
        h[2 * i] = pack_half2(__float22half2_rn(__ffma2_rn(__fadd2_rn(f01, bias2), sc2, mn2)));
        h[2 * i + 1] = pack_half2(__float22half2_rn(__ffma2_rn(__fadd2_rn(f23, bias2), sc2, mn2)));
    }
}

// The 16 weights a row's 64-weight NF4 block can hold, fp16(table[i] * absmax), as registers that byte permutes can index:
// lo[j] / hi[j] hold the low / high bytes of entries 4 j .. 4 j + 3.
struct Nf4Book {
    uint32_t lo[4], hi[4];
};
__device__ __forceinline__ void nf4_book(const float* table, float am, Nf4Book& b) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t e01 = pack_half2(__floats2half2_rn(table[4 * j] * am, table[4 * j + 1] * am));
        const uint32_t e23 = pack_half2(__floats2half2_rn(table[4 * j + 2] * am, table[4 * j + 3] * am));
        b.lo[j] = __byte_perm(e01, e23, 0x6420);
        b.hi[j] = __byte_perm(e01, e23, 0x7531);
    }
}
// Eight NF4 weights (one word, low nibble first) -> 4 fp16 pairs.  A byte permute looks up four nibbles' low three bits
// in eight entries; the nibbles' top bits choose between the results for entries 0-7 and 8-15.  No shared memory: a
// table there costs a data-dependent bank conflict per lookup (this loop took 1.2 us per step with one).
__device__ __forceinline__ void dequant_nf4(uint32_t w, const Nf4Book& b, uint32_t* h) {
    const uint32_t low3 = w & 0x77777777u, top = (w >> 3) & 0x11111111u;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t sel = low3 >> (16 * half), m = __byte_perm(0x0000ff00u, 0u, top >> (16 * half));  // 0xff where the top bit is set
        const uint32_t lo = (__byte_perm(b.lo[0], b.lo[1], sel) & ~m) | (__byte_perm(b.lo[2], b.lo[3], sel) & m);
        const uint32_t hi = (__byte_perm(b.hi[0], b.hi[1], sel) & ~m) | (__byte_perm(b.hi[2], b.hi[3], sel) & m);
        h[2 * half] = __byte_perm(lo, hi, 0x5140);
        h[2 * half + 1] = __byte_perm(lo, hi, 0x7362);
    }
}

// One instantiation per weight format: the dequantizing loop holds only its own format's code.
template <int KIND>
__global__ void __launch_bounds__(kUmmaThreads, 1)
matmul_umma_kernel(const __grid_constant__ UmmaGroup grp) {
    extern __shared__ uint8_t smem_raw[];
    uint32_t gi = 0;
#pragma unroll
    for (uint32_t i = 1; i < (uint32_t)kMaxGroup; ++i)
        if (i < grp.count && blockIdx.x >= grp.tile_start[i]) gi = i;
    const UmmaProblem& p = grp.p[gi];
    const CUtensorMap& map_w = grp.map_w[gi];
    const CUtensorMap& map_x = grp.map_x[gi];
    // full / empty of the A stages in tensor memory (quantized weights), of the operand stages in shared memory and of the
    // raw weight stages
    __shared__ uint64_t a_full[kMaxStages], a_empty[kMaxStages], b_full[kMaxStages], b_empty[kMaxStages], raw_full[kMaxRaw],
        raw_empty[kMaxRaw], done_bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ __align__(16) float code_book[16];
    __shared__ int abort_flag;

    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    constexpr bool quantized = KIND != MAT_FP16;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    // what the loops below use, in registers: read from the parameters, each would be fetched again after every asm
    // statement (several memory round trips per step)
    const uint32_t n_tile = grp.n_tile, bu = grp.bu, a_stages = grp.a_stages, b_stages = grp.b_stages, n_raw = grp.raw, splits = grp.splits;
    const uint32_t M = p.M;
    int32_t* const status = grp.status;
    const uint32_t b_step = n_tile * BK * 2, b_bytes = bu * b_step;
    constexpr uint32_t raw_row = KIND == MAT_INT8 ? 128u : 64u;  // raw bytes per row and pair of steps
    constexpr uint32_t raw_bytes = BM * raw_row;
    uint8_t* b_base = smem;                           // [b_stages] activation stages
    uint8_t* w_base = smem + b_stages * b_bytes;      // fp16: [b_stages] weight stages; else [raw] raw stages and the scales
    const uint32_t m0 = (blockIdx.x - grp.tile_start[gi]) * BM, n0 = blockIdx.y * n_tile;
    // this CTA's share of K (split-K: grid.z CTAs per output tile) in units: a pair of steps for quantized weights, a
    // stage for fp16 ones
    const uint32_t unit = quantized ? 2u : bu, units = (grp.K / BK + unit - 1) / unit;
    const uint32_t u_begin = units * blockIdx.z / splits, nu = units * (blockIdx.z + 1) / splits - u_begin;
    // the first weights are on their way before anything else is set up
    auto load_raw = [&](uint32_t u, uint32_t stage) {
        mbar_expect_tx(&raw_full[stage], raw_bytes);
        tma_load_2d(w_base + stage * raw_bytes, &map_w, (u_begin + u) * raw_row, m0, &raw_full[stage]);
    };
    auto load_weights = [&](uint32_t u, uint32_t stage) {
        mbar_expect_tx(&b_full[stage], bu * A_STEP_BYTES);
        tma_load_3d(w_base + stage * bu * A_STEP_BYTES, &map_w, 0, m0, (u_begin + u) * bu, &b_full[stage]);
    };
    const uint32_t ahead = min(nu, quantized ? n_raw : b_stages);
    uint32_t copies = 0;  // of a TMA thread: issued so far, in the order of its ring
    if (warp == kWeightTmaWarp) {
        if (elect_one()) {
            if (quantized) {
                for (uint32_t r = 0; r < n_raw; ++r) {
                    mbar_init(&raw_full[r], 1);
                    mbar_init(&raw_empty[r], kDequantWarps / 2);  // the four warps of a dequantizing group
                }
            } else {
                for (uint32_t r = 0; r < b_stages; ++r) mbar_init(&b_full[r], 2);  // both TMA threads
            }
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
#pragma unroll 1
            for (uint32_t u = 0; u < ahead; ++u) {
                if (quantized) load_raw(u, u);
                else load_weights(u, u);
            }
            copies = ahead;
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_base_slot)), "r"(grp.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    } else if (warp == kMmaWarp + 2) {
        if (elect_one()) {
            prefetch_map(&map_x);
            for (uint32_t s = 0; s < b_stages; ++s) {
                if (quantized) mbar_init(&b_full[s], 1);
                mbar_init(&b_empty[s], 1);
            }
            for (uint32_t s = 0; s < a_stages; ++s) {
                mbar_init(&a_full[s], kDequantWarps / 2);
                mbar_init(&a_empty[s], 1);
            }
            mbar_init(&done_bar, 1);
            abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
    } else if (KIND == MAT_NF4 && threadIdx.x < 16) {
        code_book[threadIdx.x] = p.table[threadIdx.x];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = tmem_base_slot, tmem_a = tmem_d + grp.acc_cols;
    // the next kernel of a job may start from here on: this CTA has its tensor memory, so neither can wait for the other's
    pdl_launch_dependents();

    if (warp < kDequantWarps) {
        if (quantized) {
            // ---- dequantizers: two groups of four warps take alternate pairs of steps (an Int8 block of 128 columns, two
            // NF4 blocks), so one group computes while the other waits; a thread owns a row, i.e. a lane of tensor memory,
            // and writes each step's 64 weights there as fp16 pairs ----
            const uint32_t group = warp >> 2, row = threadIdx.x & (BM - 1), m = m0 + row;
            const uint32_t lanes = ((warp & 3) * 32) << 16;
            // one word of scales per row and pair (Int8 (min, max), NF4 two absmax): a thread copies its own row's words into
            // its own slots of shared memory, kScaleAhead of the group's pairs before their use (a memory round trip lasts
            // longer than a pair)
            const uint32_t* srow = reinterpret_cast<const uint32_t*>(p.scale) + (size_t)(m < M ? m : 0) * (grp.K / (2 * BK));
            uint32_t* my_scale = reinterpret_cast<uint32_t*>(w_base + n_raw * raw_bytes) + group * kScaleSlots * BM + row;
            auto fetch_scale = [&](uint32_t i) {  // the group's i-th pair
                const uint32_t u = group + 2 * i;
                if (u < nu) cp_async4z(my_scale + (i % kScaleSlots) * BM, srow + u_begin + u, m < M);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            };
#pragma unroll 1
            for (uint32_t i = 0; i < kScaleAhead; ++i) fetch_scale(i);
            Ring raw, a;  // of this group's next pair
            raw.skip(group, n_raw);
            a.skip(group, a_stages);
            const uint32_t swz = KIND == MAT_INT8 ? (row & 7) : ((row >> 1) & 3);  // the TMA unit's swizzle of this row
#pragma unroll 1
            for (uint32_t u = group, i = 0; u < nu; u += 2, ++i) {
                if (u - a_stages < 2) pdl_wait();  // the group's first pair that has to wait for an MMA
                fetch_scale(i + kScaleAhead);
                asm volatile("cp.async.wait_group %0;\n" ::"n"(kScaleAhead) : "memory");
                const uint32_t sc_word = my_scale[(i % kScaleSlots) * BM];
                const float2 mm = __half22float2(*reinterpret_cast<const __half2*>(&sc_word));
                mbar_wait(&raw_full[raw.stage], raw.phase, &abort_flag, status);
                constexpr int kVecs = raw_row / 32;  // 16-byte pieces of a step
                const uint8_t* rs = w_base + raw.stage * raw_bytes + row * raw_row;
                // not unrolled: the warps of the kernel run four different loops, which together have to stay in the
                // instruction caches of their schedulers (unrolled, a fifth of all stalls waited for instructions)
#pragma unroll 1
                for (uint32_t d = 0; d < 2; ++d) {
                    uint4 q[kVecs];
#pragma unroll
                    for (uint32_t c = 0; c < kVecs; ++c) q[c] = *reinterpret_cast<const uint4*>(rs + (((kVecs * d + c) ^ swz) << 4));
                    if (d == 1) {
                        __syncwarp();  // every lane has its raw bytes in registers
                        if (lane == 0) mbar_arrive(&raw_empty[raw.stage]);
                    }
                    uint32_t h[32];
                    if (KIND == MAT_INT8) {
                        const float sc = (mm.y - mm.x) * (1.0f / 255.0f);
#pragma unroll
                        for (int c = 0; c < kVecs; ++c) dequant_int8(q[c], sc, mm.x, h + (8 * c) % 32);
                    } else {
                        Nf4Book book;
                        nf4_book(code_book, d == 0 ? mm.x : mm.y, book);
#pragma unroll
                        for (int c = 0; c < kVecs; ++c) {
                            dequant_nf4(q[c].x, book, h + (16 * c) % 32);
                            dequant_nf4(q[c].y, book, h + (16 * c) % 32 + 4);
                            dequant_nf4(q[c].z, book, h + (16 * c) % 32 + 8);
                            dequant_nf4(q[c].w, book, h + (16 * c) % 32 + 12);
                        }
                    }
                    if (d == 0) {
                        mbar_wait(&a_empty[a.stage], a.phase ^ 1, &abort_flag, status);  // at once in the stage's first use
                        tc_fence_after();
                    }
                    tmem_st32(tmem_a + lanes + (2 * a.stage + d) * A_STEP_COLS, h);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[a.stage]);
                raw.skip(2, n_raw);
                a.skip(2, a_stages);  // past the other group's pair
            }
        }
        // ---- the accumulator to shared memory, [token][128 rows] in f32 (the operand stages are free once every MMA has
        // completed): warp w holds lanes 32 (w % 4) .. and takes half of the columns ----
        pdl_wait();
        mbar_wait(&done_bar, 0, &abort_flag, status);
        tc_fence_after();
        const uint32_t quad = warp & 3, c_begin = (warp >> 2) * (n_tile / 2), c_end = c_begin + n_tile / 2;
        float* tile = reinterpret_cast<float*>(smem) + quad * 32 + lane;
#pragma unroll 1
        for (uint32_t c0 = c_begin; c0 < c_end; c0 += 32) {
            uint32_t v[4][8];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (c0 + 8 * q < c_end) tmem_ld8(tmem_d + ((quad * 32) << 16) + c0 + 8 * q, v[q]);
            tmem_ld_wait();
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                if (c0 + 8 * q >= c_end) break;
#pragma unroll
                for (int j = 0; j < 8; ++j) tile[(c0 + 8 * q + j) * BM] = __uint_as_float(v[q][j]);
            }
        }
    } else if (warp == kMmaWarp) {
        // ---- MMA issuer: one thread ----
        if (elect_one()) {
            const uint32_t idesc = f16_idesc(BM, n_tile);
            Ring ra, rb;
            pdl_wait();
            bool have_a = quantized && mbar_test(&a_full[0], 0), have_b = mbar_test(&b_full[0], 0);
            uint32_t accumulate = 0;
            // the stage of shared memory that comes next: its `steps` steps, four MMAs of K = 16 each (32 bytes of K per
            // instruction: + 2 in a descriptor's address field)
            auto stage = [&](uint32_t ta) {
                if (!have_b) mbar_wait(&b_full[rb.stage], rb.phase, &abort_flag, status);
                tc_fence_after();
                const uint64_t db = sw128_desc(smem_addr(b_base + rb.stage * b_bytes));
                const uint64_t da = quantized ? 0 : sw128_desc(smem_addr(w_base + rb.stage * bu * A_STEP_BYTES));
                uint64_t* done = &b_empty[rb.stage];
                rb.next(b_stages);
                have_b = mbar_test(&b_full[rb.stage], rb.phase);  // of the next stage: answered while this one is issued
#pragma unroll 1
                for (uint32_t d = 0; d < bu; ++d) {
#pragma unroll
                    for (uint32_t kk = 0; kk < BK / 16; ++kk) {
                        if (quantized) umma_f16_ta(tmem_d, ta + d * A_STEP_COLS + 8 * kk, db + d * (b_step >> 4) + 2 * kk, idesc, accumulate);
                        else umma_f16(tmem_d, da + d * (A_STEP_BYTES >> 4) + 2 * kk, db + d * (b_step >> 4) + 2 * kk, idesc, accumulate);
                        accumulate = 1;
                    }
                }
                umma_commit(done);  // arrives when the MMAs above have read the stage
            };
#pragma unroll 1
            for (uint32_t u = 0; u < nu; ++u) {
                if (quantized) {
                    if (!have_a) mbar_wait(&a_full[ra.stage], ra.phase, &abort_flag, status);
                    const uint32_t ta = tmem_a + 2 * ra.stage * A_STEP_COLS;
                    uint64_t* done = &a_empty[ra.stage];
                    ra.next(a_stages);
                    have_a = mbar_test(&a_full[ra.stage], ra.phase);
#pragma unroll 1
                    for (uint32_t d = 0; d < 2; d += bu) stage(ta + d * A_STEP_COLS);
                    umma_commit(done);
                } else {
                    stage(0);
                }
            }
            umma_commit(&done_bar);
        }
        __syncwarp();
    } else if (warp == kWeightTmaWarp) {
        if (elect_one()) {
            Ring ring;
            ring.skip(ahead, quantized ? n_raw : b_stages);
#pragma unroll 1
            for (uint32_t u = ahead; u < nu; ++u) {
                // a stage that is free only after an MMA: the pair before it in the ring has found no A stage unused
                if (u - ahead == (quantized ? a_stages : 0)) pdl_wait();
                if (quantized) {
                    if (!mbar_wait(&raw_empty[ring.stage], ring.phase ^ 1, &abort_flag, status)) break;
                    load_raw(u, ring.stage);
                    ring.next(n_raw);
                } else {
                    if (!mbar_wait(&b_empty[ring.stage], ring.phase ^ 1, &abort_flag, status)) break;
                    load_weights(u, ring.stage);
                    ring.next(b_stages);
                }
                copies = u + 1;
            }
        }
        __syncwarp();
    } else {
        if (elect_one()) {
            pdl_wait();  // the only loads of what a kernel before this one wrote; the outputs are stored after they have arrived
            Ring ring;
#pragma unroll 1
            for (uint32_t u = 0; u < nu; ++u) {
                const uint32_t first = (u_begin + u) * unit;
                bool ok = true;
#pragma unroll 1
                for (uint32_t d = 0; d < unit; d += bu) {
                    ok = mbar_wait(&b_empty[ring.stage], ring.phase ^ 1, &abort_flag, status);
                    if (!ok) break;
                    mbar_expect_tx(&b_full[ring.stage], b_bytes);
                    tma_load_3d(b_base + ring.stage * b_bytes, &map_x, 0, n0, first + d, &b_full[ring.stage]);
                    ring.next(b_stages);
                    ++copies;
                }
                if (!ok) break;
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    if (splits > 1) cluster_sync();  // a hardware barrier that every thread reaches, also after a wait above has given up
    else __syncthreads();
    if (copies != 0 && abort_flag != 0) {  // nobody has waited for the last copies: a thread of this CTA stays until they have landed
        const bool packed = quantized && warp == kWeightTmaWarp;
        uint64_t* const full = packed ? raw_full : b_full;
        const uint32_t stages = packed ? n_raw : b_stages;
#pragma unroll 1
        for (uint32_t j = copies - min(copies, stages); j < copies; ++j)
#pragma unroll 1
            for (uint32_t i = 0; i < kDrainLimit && !mbar_try(&full[j % stages], j / stages & 1); ++i) {
            }
    }
    if (warp == kMmaWarp) {
        if (abort_flag != 0) {  // nor for the last MMAs
#pragma unroll 1
            for (uint32_t i = 0; i < kDrainLimit && !mbar_try(&done_bar, 0); ++i) {
            }
            __syncwarp();
        }
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_d), "r"(grp.tmem_cols) : "memory");
    }
    // ---- from shared memory to the output, four rows of a token per thread and step (adjacent elements of the output).  With
    // K split over a cluster, CTA r finishes its share of the columns: the sum over its peers' tiles, through distributed
    // shared memory, in rank order (it does not depend on timing) ----
    const uint32_t rank = splits > 1 ? cluster_rank() : 0;
    const uint32_t v_lo = n_tile * rank / splits * (BM / 4), v_hi = min(n_tile * (rank + 1) / splits, grp.N - n0) * (BM / 4);
    const uint32_t tile_addr = smem_addr(smem);
    const bool out_vec = reinterpret_cast<uintptr_t>(p.out.base) % 16 == 0, f16 = p.out.dtype == WRK_F16;
    const size_t col_stride = p.out.stride[0], at0 = p.out.index(m0, n0, 0);
    const int act = p.act;
    constexpr uint32_t kBatch = 4;  // positions whose loads are in flight together
#pragma unroll 1
    for (uint32_t base = v_lo + threadIdx.x; base < v_hi; base += kBatch * kUmmaThreads) {
        float4 sum[kBatch];
#pragma unroll
        for (uint32_t i = 0; i < kBatch; ++i) sum[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (uint32_t z = 0; z < splits; ++z) {
            float4 v[kBatch];
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                const uint32_t pos = min(base + i * kUmmaThreads, v_hi - 1);
                v[i] = splits > 1 ? ld_peer_smem(tile_addr + pos * 16, z) : *reinterpret_cast<const float4*>(smem + pos * 16);
            }
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) sum[i].x += v[i].x, sum[i].y += v[i].y, sum[i].z += v[i].z, sum[i].w += v[i].w;
        }
#pragma unroll
        for (uint32_t i = 0; i < kBatch; ++i) {
            const uint32_t pos = base + i * kUmmaThreads, c = pos / (BM / 4), row = (pos % (BM / 4)) * 4;
            if (pos >= v_hi || m0 + row >= M) continue;
            const float4 r = act != WRK_ACT_NONE ? activate4(act, sum[i]) : sum[i];
            const size_t at = at0 + c * col_stride + row;
            if (m0 + row + 3 < M && (at & 3) == 0 && out_vec) {
                if (f16) {
                    const __half2 lo = __floats2half2_rn(r.x, r.y), hi = __floats2half2_rn(r.z, r.w);
                    *reinterpret_cast<uint2*>(static_cast<__half*>(p.out.base) + at) = make_uint2(pack_half2(lo), pack_half2(hi));
                } else {
                    *reinterpret_cast<float4*>(static_cast<float*>(p.out.base) + at) = r;
                }
            } else {
                dstore(p.out.base, p.out.dtype, at, r.x);
                if (m0 + row + 1 < M) dstore(p.out.base, p.out.dtype, at + 1, r.y);
                if (m0 + row + 2 < M) dstore(p.out.base, p.out.dtype, at + 2, r.z);
                if (m0 + row + 3 < M) dstore(p.out.base, p.out.dtype, at + 3, r.w);
            }
        }
    }
    if (splits > 1) cluster_sync();  // the peers have read this CTA's shared memory
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry-point lookup: the library does not link libcuda.
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

bool make_map(CUtensorMap* map, CUtensorMapDataType dt, const void* base, std::initializer_list<uint64_t> dims,
              std::initializer_list<uint64_t> strides, std::initializer_list<uint32_t> box, CUtensorMapSwizzle swz) {
    EncodeTiledFn fn = encode_tiled();
    if (fn == nullptr) return false;
    cuuint64_t gdim[3], gstride[2];
    cuuint32_t gbox[3];
    const cuuint32_t estr[3] = {1, 1, 1};
    std::copy(dims.begin(), dims.end(), gdim);
    std::copy(strides.begin(), strides.end(), gstride);
    std::copy(box.begin(), box.end(), gbox);
    return fn(map, dt, (cuuint32_t)dims.size(), const_cast<void*>(base), gdim, gstride, gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// fp16 [rows][K], rows row_bytes apart, as boxes of [steps][box_rows][64 values]: K in steps of 64 is the outermost dimension,
// so one copy brings several steps, each a tile of its own in the 128-byte swizzle
bool make_operand_map(CUtensorMap* map, const void* base, uint32_t K, uint32_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t steps) {
    return make_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, base, {BK, rows, K / BK}, {row_bytes, BK * 2}, {BK, box_rows, steps},
                    CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

bool matmul_umma_supported(const MatmulArgs& a) {
    // 9 to 15 tokens, and quantized weights of an odd number of 128-blocks, stay with the mma.sync kernel, which has them with
    // smaller errors: it multiplies Int8 bytes exactly where this one rounds each weight to fp16, and its sums lose less.
    // Relative error against float64, 12 tokens, mma.sync / this kernel: Int8 4096 x 4096 2.8e-7 / 2.0e-4, 2688 x 768 2.6e-7 /
    // 1.9e-4; NF4 2560 x 2560 1.84e-4 / 1.87e-4; fp16 4096 x 4096 6.5e-7 / 1.26e-6.
    if (a.B != 1 || a.N < 16 || a.M == 0) return false;
    if (a.K % BK != 0 || (a.kind != MAT_FP16 && a.K % (4 * BK) != 0)) return false;
    if (reinterpret_cast<uintptr_t>(a.matrix) % 16 != 0) return false;
    if (a.scale != nullptr && reinterpret_cast<uintptr_t>(a.scale) % 4 != 0) return false;
    // activations go through a tensor map: fp16, rows 16-byte aligned
    if (a.in.dtype != WRK_F16 || a.in.stride[0] % 8 != 0) return false;
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(a.in.base) + a.in.index(0, 0, 0) * 2;
    if (x0 % 16 != 0) return false;
    return encode_tiled() != nullptr;
}

// Output tiles are 128 rows x n_tile tokens; K is split across the CTAs of a thread-block cluster while the
// tiles alone leave SMs idle: a split keeps at least eight steps, a cluster at most 8 CTAs.  Up to 512 tokens,
// 128-token tiles replace 256-token ones when that doubles the CTAs of the single wave without lengthening a CTA's
// K walk: smaller operand stages (a deeper ring) and smaller partial tiles.  (Measured: 2048x2048 Int8, 256 tokens:
// 22.8 -> 15.9 us; where the K walk would double instead, 31 -> 37 us, so those keep 256.)
UmmaPlan umma_plan(int kind, uint32_t K, uint32_t N, uint32_t row_tiles, uint32_t num_sms) {
    UmmaPlan p{};
    const bool quantized = kind != MAT_FP16;
    const uint32_t nk = K / BK;
    auto splits_for = [&](uint32_t n_tile) {
        const uint64_t tiles = (uint64_t)row_tiles * ((N + n_tile - 1) / n_tile);
        uint32_t want = std::max<uint32_t>(1, (uint32_t)(num_sms / tiles));
        want = std::min<uint32_t>(want, std::max<uint32_t>(1, nk / 8));
        want = std::min<uint32_t>(want, 8);
        while (nk % 4 == 0 && nk % (4 * want) != 0) --want;  // equal shares where K allows them
        return want;
    };
    p.n_tile = std::min<uint32_t>(256, (N + 15) / 16 * 16);
    p.splits = splits_for(p.n_tile);
    if (p.n_tile > 128 && N <= 512) {
        const uint32_t s2 = splits_for(128);
        if (s2 >= p.splits && row_tiles * ((N + 127) / 128) * s2 <= num_sms) p.n_tile = 128, p.splits = s2;
    }
    // a copy of activations brings two steps unless a step's tile is large already; fewer, larger copies: issuing one costs
    // its thread about 0.2 us, as much as the MMAs of a step of 64 tokens take
    p.bu = p.n_tile <= 128 ? 2 : 1;
    // tensor memory: the accumulator and (quantized weights) A stages of a pair of steps
    p.acc_cols = (p.n_tile + 31) / 32 * 32;
    uint32_t cols = p.acc_cols;
    if (quantized) {
        cols = p.acc_cols <= 64 ? 256 : 512;
        p.a_stages = std::min<uint32_t>(kMaxStages, (cols - p.acc_cols) / (2 * A_STEP_COLS));
    }
    for (p.tmem_cols = 32; p.tmem_cols < cols;) p.tmem_cols *= 2;
    const uint32_t unit = quantized ? 2 : p.bu;
    p.walk = ((nk + unit - 1) / unit + p.splits - 1) / p.splits;
    const uint32_t b_bytes = p.bu * p.n_tile * BK * 2;
    const uint32_t raw_bytes = kind == MAT_INT8 ? BM * 128 : kind == MAT_NF4 ? BM * 64 : 0;
    const uint32_t budget = 222u * 1024;  // of an SM's shared memory: less the static part and the alignment slack
    size_t smem = 0;
    if (quantized) {
        p.b_stages = std::min<uint32_t>(kMaxStages, std::max<uint32_t>(2, p.walk * (2 / p.bu)));
        p.raw = std::min<uint32_t>(kMaxRaw, std::max<uint32_t>(2, p.walk));
        auto bytes = [&] { return p.b_stages * b_bytes + p.raw * raw_bytes + SCALE_BYTES; };
        while (bytes() > budget) {
            if (p.raw > 4) --p.raw;
            else if (p.b_stages > 4) --p.b_stages;
            else if (p.raw > 2) --p.raw;
            else --p.b_stages;
        }
        // The dequantizing groups take alternate pairs.  With an even ring a raw stage always belongs to one group, whose
        // waits see its phases in order.  With an odd one it changes hands with every use, and a group may only test it for
        // pair u when pair u - raw has arrived (a barrier two phases behind looks complete): its last pair, u - 2, waited
        // for the MMAs of pair u - 2 - a_stages, which tells it so only if raw >= a_stages + 2.
        if (p.raw < p.walk && p.raw % 2 == 1 && p.raw < p.a_stages + 2) --p.raw;
        smem = bytes();
    } else {
        const uint32_t stage = b_bytes + p.bu * A_STEP_BYTES;
        p.b_stages = std::min<uint32_t>(std::min<uint32_t>(kMaxStages, budget / stage), std::max<uint32_t>(2, p.walk));
        smem = p.b_stages * stage;
    }
    p.smem = (uint32_t)std::max<size_t>(smem, (size_t)p.n_tile * BM * sizeof(float)) + 1024;  // at the end the f32 tile lies there
    // A CTA of a cluster keeps its tensor memory until its peers have met it, and an allocation waits without limit.  Were CTAs of
    // two such launches (of two streams) to share an SM, each could wait on one SM for what the other holds on another.
    // More than half of an SM's shared memory keeps them apart.  (CTAs that are not split free theirs by themselves.)
    if (p.splits > 1) p.smem = std::max(p.smem, kSplitSmem);
    return p;
}

// The layout of a group's launch; false when its members do not go together.  Whole chunks of 32 tokens are split along K as far
// as the group's tiles leave SMs idle.  Other counts keep the sums of the single ops, bit for bit: each member's own tile and
// split have to agree, and the launch takes them.  (A group of its own splits K less, and longer sums lose more: four 2048 x 2048
// fp16 matrices at 16 tokens 1.25e-6 from float64 against 6.5e-7.)
static bool group_plan(const MatmulArgs* a, int count, uint32_t num_sms, UmmaPlan* plan) {
    if (count < 1 || count > kMaxGroup) return false;
    uint32_t row_tiles = 0;
    for (int i = 0; i < count; ++i) {
        if (!matmul_umma_supported(a[i])) return false;
        if (a[i].kind != a[0].kind || a[i].K != a[0].K || a[i].N != a[0].N) return false;
        row_tiles += (a[i].M + BM - 1) / BM;
    }
    if (a[0].N % 32 == 0) {
        *plan = umma_plan(a[0].kind, a[0].K, a[0].N, row_tiles, num_sms);
        return true;
    }
    for (int i = 0; i < count; ++i) {
        if (count > 1 && matmul_small_supported(a[i])) return false;  // alone it takes another kernel
        const UmmaPlan own = umma_plan(a[i].kind, a[i].K, a[i].N, (a[i].M + BM - 1) / BM, num_sms);
        if (i == 0) *plan = own;
        else if (own.n_tile != plan->n_tile || own.splits != plan->splits) return false;
    }
    return true;
}

bool matmul_umma_group_supported(const MatmulArgs* a, int count, int num_sms) {
    UmmaPlan plan;
    return group_plan(a, count, (uint32_t)num_sms, &plan);
}

cudaError_t matmul_umma_group(const MatmulArgs* args, int count, int32_t* status, cudaStream_t stream) {
    int sms = 148, device = 0;
    if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    UmmaPlan plan;
    if (!group_plan(args, count, (uint32_t)sms, &plan)) return cudaErrorInvalidValue;
    const MatmulArgs& a = args[0];
    UmmaGroup g{};
    g.count = (uint32_t)count;
    uint32_t row_tiles = 0;
    for (int i = 0; i < count; ++i) {
        g.tile_start[i] = row_tiles;
        row_tiles += (args[i].M + BM - 1) / BM;
    }
    for (int i = count; i <= kMaxGroup; ++i) g.tile_start[i] = row_tiles;
    g.K = a.K;
    g.N = a.N;
    g.status = status;
    g.n_tile = plan.n_tile;
    g.acc_cols = plan.acc_cols;
    g.tmem_cols = plan.tmem_cols;
    g.bu = plan.bu;
    g.a_stages = plan.a_stages;
    g.b_stages = plan.b_stages;
    g.raw = plan.raw;
    g.splits = plan.splits;

    for (int i = 0; i < count; ++i) {
        const MatmulArgs& ai = args[i];
        UmmaProblem& pi = g.p[i];
        pi.scale = ai.scale;
        pi.table = ai.table;
        pi.M = ai.M;
        pi.out = ai.out;
        pi.act = ai.act;
        bool ok;
        if (a.kind == MAT_FP16)
            ok = make_operand_map(&g.map_w[i], ai.matrix, a.K, ai.M, (uint64_t)a.K * 2, BM, g.bu);
        else if (a.kind == MAT_INT8)
            ok = make_map(&g.map_w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, ai.matrix, {a.K, ai.M}, {a.K}, {128, BM}, CU_TENSOR_MAP_SWIZZLE_128B);
        else
            ok = make_map(&g.map_w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, ai.matrix, {a.K / 2, ai.M}, {a.K / 2}, {64, BM}, CU_TENSOR_MAP_SWIZZLE_64B);
        const __half* x0 = static_cast<const __half*>(ai.in.base) + ai.in.index(0, 0, 0);
        ok = ok && make_operand_map(&g.map_x[i], x0, a.K, a.N, (uint64_t)ai.in.stride[0] * 2, g.n_tile, g.bu);
        if (!ok) return cudaErrorInvalidValue;
    }

    static SmemOptIn opt_in[3];
    auto kernel = a.kind == MAT_INT8 ? matmul_umma_kernel<MAT_INT8> : a.kind == MAT_NF4 ? matmul_umma_kernel<MAT_NF4> : matmul_umma_kernel<MAT_FP16>;
    if (cudaError_t e = opt_in[a.kind == MAT_INT8 ? 0 : a.kind == MAT_NF4 ? 1 : 2].ensure(kernel, 223 * 1024); e != cudaSuccess) return e;
    dim3 grid(row_tiles, (a.N + g.n_tile - 1) / g.n_tile, g.splits);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kUmmaThreads, 1, 1);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = g.splits;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained_launches() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, g);
}

cudaError_t matmul_umma(const MatmulArgs& a, int32_t* status, cudaStream_t stream) { return matmul_umma_group(&a, 1, status, stream); }

}  // namespace k
}  // namespace wrk
