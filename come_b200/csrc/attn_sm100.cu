// Variable-length biased attention forward on Blackwell tensor cores (sm_100a): tcgen05.mma with TMEM
// accumulators, TMA-fed 128-byte-swizzled Q/K/V tiles, warp-specialised roles.
//
// Persistent kernel: one CTA per SM walks the work items; a work item is one to four 128-row query tiles of one
// (segment, head), whose keys are walked 64 at a time.  Barrier phases keep counting across items.
//   warps 0-15     : softmax groups of query tiles 0 .. 3, four warps each.  Thread r owns score row r (TMEM lane r).  Per key
//                     tile it pulls the 64 scores into registers, takes the row max with 3-input max, then
//                     p = exp2(s * scale*log2e - m) in packed float32x2 arithmetic, a share of the exponentials on the FMA
//                     pipe (cubic polynomial) instead of the special-function unit, writes p over the first half of its
//                     scores as 16-bit pairs (the A operand of P V) and rescales the accumulator only when the running max
//                     grew by more than 2^8 (exact: the final normalisation uses the same reference max).
//   warp 16         : producer.  Issues the TMA loads of Q (double-buffered across items), K and V and stages, per key
//                     tile, a "bias slab": a 64 x 16 tile whose first two columns hold bias/scale split into a high and a
//                     low 16-bit part (a large negative number past the segment end, which masks the ragged tail).
//   warps 17, 18    : MMA issuers of query tiles 0, 2 / 1, 3.  When P(j) of a tile is staged they issue O += P(j) V(j), with P
//                     from TMEM and V (N-major) from shared memory, and right behind it S = Q K(j+1)^T over the same columns
//                     (four K=16 steps over the head dimension plus one K=16 step [1 1 0 ...] x [bias_hi bias_lo 0 ...]^T that
//                     adds the per-key bias inside the tensor core).  ONE barrier per tile and direction then carries a key
//                     step: "P staged" and "scores complete", which also says that the accumulator is stable.
// TMEM columns: S_t / P_t [64 t, 64 t + 64), O_t [256 + 64 t, ...), t = 0 .. 3.
//
// P over S rests on an order that is practice, not documentation: the scores S(j+1) are written over the columns of P(j) by
// an instruction of the same thread behind the P V that reads them, with no barrier between.  PTX documents an implicit order
// for tcgen05.mma instructions of one accumulator and shape, and a commit for everything before it; these two have different
// accumulators.  The tensor pipe is taken to run the instructions of a thread in the order of issue.  An overtaking write
// would change the result from launch to launch: the tests compare bits over the number of CTAs and the query tiles per
// item (test_item_heights), over row slices, and values with the fp32 oracle.
//
// What bounds it: a key step of four tiles is ~2500 clocks (80,672 keys, 869 TFLOP/s): ~1660 of the special-function unit (13 of
// 16 exponentials of 32,768, 16 per clock), ~1600 issue slots per scheduler, ~1470 of the tensor pipe (an M128 N64 K16
// instruction with both operands in shared memory takes 48 clocks, with P in tensor memory 32).  No unit is full: a tile
// alone takes ~1500 (softmax 850, hand-over and issue 260, tensor work 370), its chain is serial, and four tiles overlap.  The
// nine instructions of a tile and step are issued in ~190 clocks because shared-memory and tensor-memory addresses are known
// at link time, each issuer has its own copy of the code, and no wait steers its loop but for a vote every 32 key tiles; with
// operands moved from ordinary registers they took ~590.
//
// Every wait on an mbarrier is bounded: after ~2^29 clock ticks the waiter raises the CTA's abort flag and the library's
// device status word.  From then on no role acts on data it did not wait for: the producer loads and an issuer issues
// nothing more, and a softmax group stores an item only if the last P V of it was issued and has completed, so a row of the
// result is either right or untouched.  Every role falls through to the common exit, where the producer waits for its own
// loads and the issuers for their own tensor-core work (both complete by themselves; bounded all the same); then TMEM is
// released and the kernel returns instead of hanging.
#include "attn_sm100.cuh"

#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace come {

namespace {

constexpr int kTiles = 4;         // query tile slots (128 rows each) per CTA, one softmax warpgroup each
constexpr int kBlockM = 128;
constexpr int kBlockN = 64;       // keys per step
constexpr int kHeadDim = 64;
constexpr int kStages = 4;        // key tile ring: K, V (8 KiB each) and the bias slab of a key tile share a stage
constexpr int kProducerWarp = 4 * kTiles;      // warps 0 .. 4*kTiles-1 are the softmax groups
constexpr int kIssuers = 2;       // warps that issue the tensor-core work, two query tiles each
constexpr int kIssuerWarp0 = kProducerWarp + 1;
constexpr int kThreads = 32 * (kProducerWarp + 4);  // 640: four softmax warpgroups + one with the producer, the issuers and an idle warp
static_assert(kTiles % kIssuers == 0 && 1 + kIssuers <= 4, "one warpgroup holds the producer and the issuers");
// Launches with this many segments keep a prefix table of their query blocks in shared memory; with fewer, a sorted list
constexpr int kMinPrefixSegs = 16, kMaxPrefixSegs = 2048, kMaxListSegs = kMinPrefixSegs - 1;
constexpr int kQTileBytes = kBlockM * kHeadDim * 2;   // 16384
constexpr int kKvTileBytes = kBlockN * kHeadDim * 2;  // 8192
constexpr int kQSlabBytes = kBlockM * 16 * 2, kSlabBytes = kBlockN * 16 * 2;  // 16 columns of 16 bits
// Tensor-memory columns: S_t (scores, float32), whose first half P_t (probabilities, 16-bit pairs) reuses | O_t (accumulator, float32)
constexpr uint32_t kTmemS = 0, kTmemO = kTiles * kBlockN;
static_assert(kTmemO + kTiles * kHeadDim <= 512, "tensor memory holds 512 columns");
static_assert(kThreads % 128 == 0, "setmaxnreg works on whole warpgroups");
constexpr uint32_t kTmemCols = 512;
constexpr long long kWaitTicks = 1ll << 29;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f;  // log2 units
// Which of the 16 score pairs of a 32-column half take the polynomial exp2 (bit i = pair i); the rest use the
// special-function unit.  0 / 3 / 4 / 5 of 16 on the polynomial route: 828 / 839 / 827 / 810 TFLOP/s at 24,576 keys, 624 / 666 /
// 671 / 654 on 8 x 1374; the fewer take it, the less the kernel draws under the power cap.
#ifndef COME_POLY_MASK
#define COME_POLY_MASK 0x2108u
#endif
constexpr uint32_t kPolyPairs = COME_POLY_MASK;
constexpr float kMasked = -3.0e38f;        // "minus infinity" of a masked key, still finite in bfloat16

struct SharedStorage {
    alignas(1024) uint8_t q[2][kTiles][kQTileBytes];        // [buffer][query tile]: the next item's Q is loaded ahead
    alignas(1024) uint8_t k[kStages][kKvTileBytes];
    alignas(1024) uint8_t v[kStages][kKvTileBytes];
    alignas(128) uint8_t q_slab[kQSlabBytes];               // columns 0,1 = 1.0, rest 0: the A side of the bias step
    alignas(128) uint8_t k_slab[kStages][kSlabBytes];       // columns 0,1 = bias/scale (hi, lo), rest 0: the B side
    alignas(8) uint64_t q_full[2];
    uint64_t q_empty[2];
    uint64_t kv_full[kStages];
    uint64_t kv_empty[kStages];
    uint64_t q_slab_full;
    uint64_t s_full[kTiles];  // scores of a key tile complete (and, in order before them, P V of the key tile before)
    uint64_t p_full[kTiles];
    uint64_t o_done[kTiles];  // the last P V of an item complete
    uint64_t drained;         // all tensor-core work of the CTA complete (exit path)
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
    // work list (see plan_work)
    int4 seg_rows[kMaxListSegs];            // keys [x, y) and query rows [z, w) of a segment, by falling number of keys
    int4 seg_items[kTiles][kMaxListSegs];   // [height - 1]: first item of the segment, items per head, their reciprocal
    int4 plan[kTiles];                      // [height - 1]: items, first item of a split last round, its parts, their reciprocal
    float plan_cost[kTiles];
    uint32_t per_head_rcp;
    int scan_warp[kThreads / 32], sum_items[kTiles][kThreads / 32];
    float sum_cost[kTiles][kThreads / 32];
};
// Launches that use the prefix table get (kMaxPrefixSegs + 1) ints of dynamic shared memory behind SharedStorage:
// table[s] = query blocks of the segments before s (this launch's rows).
constexpr size_t kPrefixTableBytes = sizeof(int) * (kMaxPrefixSegs + 1);

static_assert(sizeof(SharedStorage) + kPrefixTableBytes + 1024 <= 227 * 1024, "shared storage exceeds the 227 KB a CTA may use");

// ---- PTX wrappers ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false (and raises the abort flag + the device status word) when it gives up after `limit`
// clock ticks, or when another waiter of the CTA has given up.
__device__ __forceinline__ bool mbar_wait_limit(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag,
                                                unsigned int *status, uint32_t code, long long limit) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag != 0) return false;
        if (clock64() - t0 > limit) {
            *abort_flag = 1;
            atomicOr(status, code);
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, SharedStorage &sh, unsigned int *status,
                                          uint32_t code) {
    return mbar_wait_limit(bar, parity, &sh.abort_flag, status, code, kWaitTicks);
}
// Bounded wait of the exit path, for work of this CTA that completes by itself: it goes on after the abort flag is raised.
__device__ __forceinline__ void mbar_drain(uint64_t *bar, uint32_t parity, unsigned int *status, uint32_t code) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > kWaitTicks) {
            atomicOr(status, code);
            return;
        }
    }
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int c0, int c1, int c2, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The issuer warps run their loops in warp-uniform control flow; for a group of instructions (the Q K^T of a key tile
// with its commits, or its P V) one lane is elected once and issues the whole group.  Electing per instruction (every
// lane evaluating the operands, one lane executing) measured 3-5 % slower: an issuer warp shares its scheduler with
// four softmax warps, and every instruction it does not issue shortens the time from "P is staged" to "P V is queued".
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
__device__ __forceinline__ void tc_commit_1(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_mma_ss_1(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_mma_ts_1(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives lane (base lane + i).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Makes generic-proxy shared-memory writes of this thread visible to the async proxy (tcgen05.mma operands).
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// The bias slabs are K-major tiles without swizzle: 8-row x 16-byte core matrices, those of columns 0..7 first (8-row
// groups 128 bytes apart), then those of columns 8..15.  Only columns 0 and 1 carry values; the rest stays zero.
__device__ __forceinline__ uint32_t slab_offset(int r) { return (uint32_t)((r >> 3) * 128 + (r & 7) * 16); }
__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t x) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}
__device__ __forceinline__ uint64_t make_slab_desc(uint32_t saddr, int rows) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);  // start address
    d |= (uint64_t)(rows) << 16;              // leading byte offset: columns 0..7 to columns 8..15, rows * 16 bytes (in units of 16)
    d |= (uint64_t)(128 >> 4) << 32;          // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                   // descriptor version of sm_100; no swizzle
    return d;
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 2^x for two values on the FMA / integer pipes instead of the special-function unit (which is the bottleneck of
// the head_dim-64 kernel): round-to-nearest range reduction x = n + f, f in [-0.5, 0.5], cubic fit of 2^f (relative
// error 1.0e-4, far below the 16-bit rounding of the probabilities), n added to the exponent field as an integer.
// Inputs below -125 are clamped (the result is then ~2^-125, i.e. zero for all purposes).
__device__ __forceinline__ void exp2_poly_x2(float x0, float x1, float &r0, float &r1) {
    const f32x2_t magic = pack_f32x2(12582912.0f, 12582912.0f);  // 1.5 * 2^23: adding it rounds to an integer
    const f32x2_t neg_magic = pack_f32x2(-12582912.0f, -12582912.0f);
    const f32x2_t minus_one = pack_f32x2(-1.0f, -1.0f);
    const f32x2_t c3 = pack_f32x2(0.05583828315138817f, 0.05583828315138817f);
    const f32x2_t c2 = pack_f32x2(0.2426394820213318f, 0.2426394820213318f);
    const f32x2_t c1 = pack_f32x2(0.6931367516517639f, 0.6931367516517639f);
    const f32x2_t c0 = pack_f32x2(0.9999245405197144f, 0.9999245405197144f);
    const f32x2_t x = pack_f32x2(fmaxf(x0, -125.0f), fmaxf(x1, -125.0f));
    const f32x2_t t = add_f32x2(x, magic);        // low mantissa bits of t hold n = round(x)
    const f32x2_t n = add_f32x2(t, neg_magic);
    const f32x2_t f = fma_f32x2(n, minus_one, x);
    f32x2_t p = fma_f32x2(c3, f, c2);
    p = fma_f32x2(p, f, c1);
    p = fma_f32x2(p, f, c0);
    float p0, p1, t0, t1;
    unpack_f32x2(p, p0, p1);
    unpack_f32x2(t, t0, t1);
    r0 = __int_as_float(__float_as_int(p0) + (__float_as_int(t0) << 23));
    r1 = __int_as_float(__float_as_int(p1) + (__float_as_int(t1) << 23));
}

template <bool kBF16> __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    if constexpr (kBF16) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t *>(&v);
    } else {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t *>(&v);
    }
}

// Multiplies the 64 float32 accumulator columns of this thread's row by alpha (the rare rescale when a row's running
// max grew past the threshold), 16 columns at a time: the scores of the key tile stay in registers meanwhile.
__device__ __forceinline__ void scale_accumulator(uint32_t o_tmem, float alpha) {
#pragma unroll 1
    for (int c = 0; c < kHeadDim; c += 16) {
        uint32_t o[16];
        tmem_ld16(o_tmem + c, o);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
        tmem_st16(o_tmem + c, o);
    }
}

// Shared-memory matrix descriptor of a tile whose rows are 128 bytes wide and 128-byte swizzled (what a TMA
// load with a 64-element 16-bit inner box produces): 8-row groups are 1024 bytes apart.  The same encoding
// serves a K-major operand (rows = M/N index, advance 32 bytes per 16-element K step) and an MN-major operand
// (rows = K index, advance 2048 bytes per 16-row K step).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);  // start address
    d |= (uint64_t)1 << 16;                   // leading byte offset (unused for a single swizzle atom)
    d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                   // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                   // 128-byte swizzle
    return d;
}

// Instruction descriptor of tcgen05.mma.kind::f16: float32 accumulate, 16-bit A/B of the given format.
__host__ __device__ constexpr uint32_t make_idesc(bool bf16, int M, int N, bool b_mn_major) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((b_mn_major ? 1u : 0u) << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

enum : uint32_t {
    kErrQFull = 1u << 0, kErrKvFull = 1u << 1, kErrKvEmpty = 1u << 2,
    kErrSFull = 1u << 5, kErrPFull = 1u << 7, kErrODone = 1u << 8, kErrTmem = 1u << 9,
    kErrSelfTest = 1u << 15,  // raised by the wait self-test on purpose
};
static_assert(((kErrQFull | kErrKvFull | kErrKvEmpty | kErrSFull | kErrPFull | kErrODone | kErrTmem) & ~kStatusAttention) == 0,
              "come_device_status names these bits");

// One work item = up to `tiles` 128-row query tiles [q_row0, q_row0 + tiles * 128) of one (segment, head).
struct WorkItem {
    int head, s0, s1;   // head, key range of the segment
    int q_row0, q_hi;   // first query row of the item, end of the query rows this launch owns in the segment
    int n_mt, n_kv;     // active query tiles (1 .. kTiles), key tiles
    int t0;             // tile slot of the first of them: items of one tile take the slots in turn, others begin at 0
    bool ragged_tail;   // the last key tile is partial
    bool valid;
    int kpart;          // which share of the keys this item covers (launches that split the keys of their items), else 0
};

__host__ __device__ constexpr int tiles_of(int rows) { return rows > 0 ? (rows + kBlockM - 1) / kBlockM : 0; }
__host__ __device__ constexpr int key_tiles_of(int keys) { return keys > 0 ? (keys + kBlockN - 1) / kBlockN : 0; }

// n / d and the remainder by the reciprocal floor((2^32 - 1) / d), for any 32-bit n: the estimate is at most one too small.
__device__ __forceinline__ uint32_t reciprocal(int d) { return d > 0 ? 0xffffffffu / (uint32_t)d : 0u; }
__device__ __forceinline__ int div_by(int n, int d, uint32_t rcp, int &rem) {
    int q = (int)__umulhi((uint32_t)n, rcp);
    rem = n - q * d;
    if (rem >= d) {
        ++q;
        rem -= d;
    }
    return q;
}

// Query tiles per work item.  A key step of an item costs less than in proportion to its tiles (the tiles share the SM's
// units but each is a latency chain: 0.79 / 0.90 / 1.06 / 1.29 us with 1 / 2 / 3 / 4 tiles, 6456 keys), so four tiles are
// best where there are many items; but the items are dealt to the CTAs in rounds, and with few of them the height that
// fills its last round wins: 6456 tokens x 16 heads take 215 us with 3 (272 items, 2 rounds) and 260 with 4 (208 items, also
// 2 rounds); 3228 tokens 59 and 68 us; 2 segments of ~450 tokens 12.0 us with 1 and 16.8 with 4; 4 x 807 tokens 24 us with
// 4 and 37 with 3.  The choice is the height with the least sum, over the rounds, of the mean cost of an item of the segment the
// round begins in (its step by its key tiles); the items of a partial last round are split into lower ones where the CTAs
// suffice for that (tail_height): 24,576 tokens x 16 heads are 768 items = 5 rounds + 28 items of four tiles, which run as 112
// items of one (3.02 -> 2.87 ms); 80,672 tokens are 17 rounds + 12 items (30.6 -> 29.7 ms).  The step costs were measured at
// 6456 keys; what an item costs beyond its steps is not in them.
__host__ __device__ __forceinline__ int step_cost(int n) { return n <= 0 ? 0 : n == 1 ? 70 : n == 2 ? 80 : n == 3 ? 96 : 115; }
// Height of the items of the last, partial round of `rest` items of `height` tiles.
__host__ __device__ __forceinline__ int tail_height(int height, int rest, int ctas) {
    if (height > 1 && rest * height <= ctas) return 1;
    if (height > 2 && rest * 2 <= ctas) return 2;
    return height;
}
__host__ __device__ __forceinline__ int blocks_of(int n, int height) {  // items of n query tiles
    return height == 1 ? n : height == 2 ? (n + 1) >> 1 : height == 4 ? (n + 3) >> 2 : (n + 2) / 3;
}
__host__ __device__ __forceinline__ int height_cost(int n, int height) {  // of these items
    const int blocks = blocks_of(n, height), rest = n - (blocks - 1) * height;
    return n <= 0 ? 0 : (blocks - 1) * step_cost(height) + step_cost(rest);
}

// Work list of a launch: the items [0, total) of `height` query tiles, of which those from `from` on are split into `parts`
// lower ones, and how an item becomes rows of a segment and a head.  Planned on the host where it knows enough, else by every
// CTA for itself.
//  * One segment, launches in which every query tile gets a CTA of its own or no segment has a second one (height 1), and
//    those with more segments than the prefix table holds: planned on the host.  `slots` blocks for every (segment, head); those beyond a
//    segment's end are skipped as invalid.
//  * 2 .. kMaxListSegs segments (the sorted list): the items are exactly those that exist, in the order (segment by falling
//    number of keys, head, block).  Dealt round-robin the CTAs then get items of like length in every round and the short ones
//    fill up at the end.  One slot per segment and maximal block in the order (head, segment, block) costs segments of unlike
//    length up to 2.7 x: 12000 + 6000 + 3000 + 1500 + 750 + 375 tokens x 6 heads took 1349 us (the long segment's blocks
//    of all heads fall on the same CTAs) and take 350; 20000 + 10 x 500 tokens x 16 heads 3817 and 1908.
//  * kMinPrefixSegs .. kMaxPrefixSegs segments (the prefix table): the items that exist in the order (head, segment, block).
// Warps 0 .. kTiles - 1 plan one height each while other warps initialise the barriers and allocate tensor memory; after the
// barrier every thread picks the cheapest.  What a short launch feels is the code that runs once, at 4 to 5 clocks per
// instruction: planned by every warp for itself, in each other's issue slots, the same took 3250 clocks.
struct WorkPlan {
    int height;  // 0: planned on the device
    int total, from, parts, slots;
    uint32_t parts_rcp, slots_rcp, nseg_rcp, ctas_rcp;
};
struct WorkArgs {
    const int *cu;        // may be NULL for q_free: [0, kv_total]
    int nseg, num_heads, q_begin, q_end, kv_total, max_rows, k_parts, ctas;
    bool q_free;
};

// Cost of a plan of `height` whose rounds cost `cost`, of which the last, partial one has `rest` items of `mean` cost and
// `keys` key tiles: its items are split into lower ones where the CTAs suffice.
__host__ __device__ __forceinline__ float split_last_round(WorkPlan &pl, int height, int items, int rest, float cost, float mean, float keys, int ctas) {
    pl.height = height;
    pl.total = pl.from = items;
    pl.parts = 1;
    pl.parts_rcp = 0xffffffffu;
    const int low = tail_height(height, rest, ctas);
    if (rest > 0 && low != height) {
        pl.parts = low == 2 ? 2 : height;
        pl.parts_rcp = pl.parts == 2 ? 0x7fffffffu : pl.parts == 3 ? 0x55555555u : 0x3fffffffu;
        pl.from = items - rest;
        pl.total = pl.from + rest * pl.parts;
        cost += (float)step_cost(low) * keys - mean;
    }
    return cost;
}
__device__ __forceinline__ void store_plan(SharedStorage &sh, const WorkPlan &pl, float cost) {
    sh.plan[pl.height - 1] = make_int4(pl.total, pl.from, pl.parts, (int)pl.parts_rcp);
    sh.plan_cost[pl.height - 1] = cost;
}

// The sorted list for items of `height` tiles, by one warp: a lane per segment.
__device__ __forceinline__ void plan_list(SharedStorage &sh, const WorkArgs &a, const WorkPlan &host, int height, int lane) {
    int4 rows = make_int4(0, 0, 0, 0);
    if (lane < a.nseg) {
        rows.x = a.cu[lane];
        rows.y = a.cu[lane + 1];
        rows.z = max(rows.x, a.q_begin);
        rows.w = min(rows.y, a.q_end);
    }
    const int keys = key_tiles_of(rows.y - rows.x), n = tiles_of(min(rows.w - rows.z, a.max_rows));
    const int blocks = blocks_of(n, height);
    int rank = 0, first = 0;
#pragma unroll 1
    for (int j = 0; j < a.nseg; ++j) {
        const int other_keys = __shfl_sync(0xffffffffu, keys, j), other_blocks = __shfl_sync(0xffffffffu, blocks, j);
        const bool before = other_keys > keys || (other_keys == keys && j < lane);
        rank += before ? 1 : 0;
        first += before ? other_blocks : 0;
    }
    first *= a.num_heads;
    const int end = first + blocks * a.num_heads;
    if (lane < a.nseg) {
        if (height == kTiles) sh.seg_rows[rank] = rows;
        sh.seg_items[height - 1][rank] = make_int4(first, blocks, (int)reciprocal(blocks), 0);
    }
    int rem;
    const int rounds_before = div_by(first + a.ctas - 1, a.ctas, host.ctas_rcp, rem);  // rounds that begin in front of the segment
    const int rounds = div_by(end + a.ctas - 1, a.ctas, host.ctas_rcp, rem) - rounds_before;
    const float mean = blocks > 0 ? __fdividef((float)height_cost(n, height), (float)blocks) * (float)keys : 0.0f;
    float cost = (float)rounds * mean;
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) cost += __shfl_xor_sync(0xffffffffu, cost, d);  // lanes 0 .. 15
    const int items = (int)__reduce_max_sync(0xffffffffu, (unsigned)end);
    int rest;
    div_by(items, a.ctas, host.ctas_rcp, rest);
    const unsigned owner = __ballot_sync(0xffffffffu, first <= items - rest && items - rest < end);
    const int src = max(__ffs(owner) - 1, 0);
    const float last = __shfl_sync(0xffffffffu, mean, src);
    const int last_keys = __shfl_sync(0xffffffffu, keys, src);
    if (lane == 0) {
        WorkPlan pl;
        cost = split_last_round(pl, height, items, rest, cost, last, (float)last_keys, a.ctas);
        store_plan(sh, pl, cost);
    }
}

__device__ __forceinline__ int cheapest_height(const SharedStorage &sh) {  // the greatest of equally cheap ones
    int height = kTiles;
    float least = sh.plan_cost[kTiles - 1];
#pragma unroll
    for (int h = kTiles - 1; h >= 1; --h) {
        const float cost = sh.plan_cost[h - 1];
        if (cost < least) {
            least = cost;
            height = h;
        }
    }
    return height;
}

// The prefix table, by the whole CTA: a height from the sums over all segments, then a scan of the query blocks.  The sums
// are formed in a fixed order, so that every CTA makes the same choice.  Returns the height.
__device__ __forceinline__ int plan_prefix(SharedStorage &sh, const WorkArgs &a, const WorkPlan &host, int *prefix) {
    constexpr int kPer = (kMaxPrefixSegs + kThreads) / kThreads;  // consecutive segments per thread
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int local[kPer], items[kTiles] = {};
    float cost[kTiles] = {};
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int sg = threadIdx.x * kPer + i;
        local[i] = 0;
        if (sg < a.nseg) {
            const int s0 = a.cu[sg], s1 = a.cu[sg + 1];
            local[i] = tiles_of(min(s1, a.q_end) - max(s0, a.q_begin));
            const float keys = (float)key_tiles_of(s1 - s0);
#pragma unroll
            for (int h = 1; h <= kTiles; ++h) {
                items[h - 1] += blocks_of(local[i], h);
                cost[h - 1] += keys * (float)height_cost(local[i], h);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < kTiles; ++h) {
        items[h] = (int)__reduce_add_sync(0xffffffffu, (unsigned)items[h]);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) cost[h] += __shfl_xor_sync(0xffffffffu, cost[h], d);
        if (lane == 0) {
            sh.sum_items[h][warp] = items[h];
            sh.sum_cost[h][warp] = cost[h];
        }
    }
    __syncthreads();
    if (warp < kTiles) {
        const bool has = lane < kThreads / 32;
        const int total = a.num_heads * (int)__reduce_add_sync(0xffffffffu, has ? (unsigned)sh.sum_items[warp][lane] : 0u);
        float sum = has ? sh.sum_cost[warp][lane] : 0.0f;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if (lane == 0) {
            const float mean = sum * (float)a.num_heads / (float)max(total, 1);
            int rest;
            int rounds = div_by(total, a.ctas, host.ctas_rcp, rest);
            rounds += rest > 0 ? 1 : 0;
            WorkPlan pl;
            const float all = split_last_round(pl, warp + 1, total, rest, (float)rounds * mean, mean, mean / (float)step_cost(warp + 1), a.ctas);
            store_plan(sh, pl, all);
        }
    }
    __syncthreads();
    const int height = cheapest_height(sh);
    int sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        local[i] = blocks_of(local[i], height);
        sum += local[i];
    }
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) sh.scan_warp[warp] = incl;
    __syncthreads();
    int before = incl - sum;
    for (int wq = 0; wq < warp; ++wq) before += sh.scan_warp[wq];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int sg = threadIdx.x * kPer + i;
        if (sg <= a.nseg) prefix[sg] = before;
        if (sg == a.nseg) sh.per_head_rcp = reciprocal(before);
        before += local[i];
    }
    return height;
}

// Plans the launch; after the caller's next __syncthreads picked_height names the height.  Returns that of a table launch.
template <bool kPrefix>
__device__ __forceinline__ int plan_work(SharedStorage &sh, const WorkArgs &a, const WorkPlan &host, int *prefix) {
    if constexpr (kPrefix) {
        return plan_prefix(sh, a, host, prefix);
    } else {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (host.height == 0) {
            if (warp < kTiles) plan_list(sh, a, host, warp + 1, lane);
        } else if (threadIdx.x == 0) {
            store_plan(sh, host, 0.0f);
            if (a.nseg == 1) {
                const int s0 = a.cu ? a.cu[0] : 0, s1 = a.cu ? a.cu[1] : a.kv_total;
                sh.seg_rows[0] = make_int4(s0, s1, a.q_free ? a.q_begin : max(s0, a.q_begin), a.q_free ? a.q_end : min(s1, a.q_end));
            }
        }
        return 0;
    }
}
__device__ __forceinline__ int picked_height(const SharedStorage &sh, int planned, const WorkPlan &host) {
    return planned != 0 ? planned : host.height != 0 ? host.height : cheapest_height(sh);
}

// Item -> (head, segment, query block), by a converged warp.
// q_free: the launch has one segment whose keys all query rows [q_begin, q_end) attend to, whether or not those rows lie
// inside the segment (attention of this GPU's rows to keys gathered from other GPUs); cu may then be NULL = [0, kv_total].
template <bool kPrefix>
__device__ __forceinline__ WorkItem decode_item(int item, const SharedStorage &sh, const WorkArgs &a, const WorkPlan &host, const int *prefix,
                                                int height) {
    WorkItem w;
    int bx, q_lo;
    w.t0 = 0;
    if (height == 1) {  // the round of the item
        int cta;
        w.t0 = div_by(item, a.ctas, host.ctas_rcp, cta) % kTiles;
    }
    int first_tile = 0, most_tiles = height;  // of the item's rows inside its block of `height` tiles
    const int4 pl = sh.plan[height - 1];
    if (item >= pl.y) {
        const int i = div_by(item - pl.y, pl.z, (uint32_t)pl.w, first_tile);
        item = pl.y + i;
        most_tiles = pl.z == height ? 1 : 2;
        first_tile *= most_tiles;
    }
    // Launches with k_parts > 1 (q_free only): consecutive items are the shares of the key tiles of one (head, block); every
    // share writes its own output and log-sum-exp, merged afterwards.  The host picks k_parts so that no share is empty.
    w.kpart = 0;
    if (a.k_parts > 1) {
        w.kpart = item % a.k_parts;
        item /= a.k_parts;
    }
    // Query rows of this launch: global rows [q_begin, q_end) (the whole packed sequence for plain self-attention; a
    // slice when the query rows are sharded).  q / out / lse are indexed by (global row - q_begin); k / v by global row.
    if constexpr (kPrefix) {
        int r;
        w.head = div_by(item, prefix[a.nseg], sh.per_head_rcp, r);
        int lo = 0, hi = a.nseg;  // last segment whose prefix is <= r
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid] <= r) lo = mid;
            else hi = mid;
        }
        bx = r - prefix[lo];
        w.s0 = a.cu[lo];
        w.s1 = a.cu[lo + 1];
        q_lo = max(w.s0, a.q_begin);
        w.q_hi = min(w.s1, a.q_end);
    } else if (host.height == 0 || a.nseg == 1) {
        int rank = 0;
        if (host.height == 0) {  // the last segment whose first item is not behind this one
            const int lane = threadIdx.x & 31;
            const int4 *list = sh.seg_items[height - 1];
            rank = __popc(__ballot_sync(0xffffffffu, lane < a.nseg && list[min(lane, kMaxListSegs - 1)].x <= item)) - 1;
            const int4 it = list[rank];
            w.head = div_by(item - it.x, it.y, (uint32_t)it.z, bx);
        } else {
            w.head = div_by(item, host.slots, host.slots_rcp, bx);
        }
        const int4 rows = sh.seg_rows[rank];
        w.s0 = rows.x;
        w.s1 = rows.y;
        q_lo = rows.z;
        w.q_hi = rows.w;
    } else {
        int seg;
        w.head = div_by(div_by(item, host.slots, host.slots_rcp, bx), a.nseg, host.nseg_rcp, seg);
        w.s0 = a.cu[seg];
        w.s1 = a.cu[seg + 1];
        q_lo = max(w.s0, a.q_begin);
        w.q_hi = min(w.s1, a.q_end);
    }
    const int seg_len = w.s1 - w.s0;
    w.q_row0 = q_lo + (bx * height + first_tile) * kBlockM;
    const int rows = min(w.q_hi - w.q_row0, min(height - first_tile, most_tiles) * kBlockM);  // of the item
    w.valid = rows > 0;
    w.n_mt = (rows + kBlockM - 1) / kBlockM;  // query tiles with at least one valid row
    w.n_kv = (seg_len + kBlockN - 1) / kBlockN;
    w.ragged_tail = (seg_len % kBlockN) != 0;
    if (a.k_parts > 1) {
        const int per_part = (w.n_kv + a.k_parts - 1) / a.k_parts;
        const int t0 = w.kpart * per_part, t1 = min(w.n_kv, t0 + per_part);
        if (t0 >= t1) {
            w.valid = false;
        } else {
            const int s0 = w.s0;
            w.s0 = s0 + t0 * kBlockN;
            w.s1 = min(w.s1, s0 + t1 * kBlockN);
            w.n_kv = t1 - t0;
            w.ragged_tail = ((w.s1 - w.s0) % kBlockN) != 0;
        }
    }
    return w;
}

// Persistent kernel: one CTA per SM walks the work items item = blockIdx.x, blockIdx.x + gridDim.x, ...  Every role
// runs the same item loop on its own; the barriers' phases simply keep counting across items, so the producer
// streams the next item's K/V and Q (two buffers of Q) while the softmax groups are still finishing the current one.
// kPrefix selects the work list at compile time, so that launches with few segments carry none of the table's code.
// kSelfTest: the producer loads the key tiles before the CTA's tile `stall_tile` only, so that the waits for that tile run out.
template <bool kBF16, bool kPrefix, bool kSelfTest = false>
__global__ void __launch_bounds__(kThreads, 1)
attn_fwd_sm100_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const void *__restrict__ bias_ptr,
                      const int *__restrict__ cu, float scale_log2, float inv_scale, void *__restrict__ out_ptr, int64_t o_rs,
                      float *__restrict__ lse, int q_begin, int q_end, int max_rows, int nseg, int num_heads,
                      const int *__restrict__ max_len_dev, unsigned int *__restrict__ status, int kv_total, int q_free_flag,
                      int k_parts, long long part_o, long long part_l, const WorkPlan host_plan, int stall_tile) {
    using T = typename std::conditional<kBF16, __nv_bfloat16, __half>::type;
    // the declared alignment makes the base, and with it every barrier address and matrix descriptor, a link-time constant
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    SharedStorage &sh = *reinterpret_cast<SharedStorage *>(smem_raw);

    // `max_rows` is the host's upper bound of the query rows of a segment.  A caller that cannot read the true length back
    // (a captured graph serving every merge mask) passes a loose bound plus the true one in device memory.
    WorkArgs work{cu, nseg, num_heads, q_begin, q_end, kv_total, max_rows, k_parts, (int)gridDim.x, q_free_flag != 0};
    if (max_len_dev != nullptr) work.max_rows = min(max_rows, max(*max_len_dev, 0));
    int *prefix = reinterpret_cast<int *>(reinterpret_cast<uint8_t *>(&sh) + sizeof(SharedStorage));  // launches with the table
    const int planned = plan_work<kPrefix>(sh, work, host_plan, prefix);
    const bool has_bias = bias_ptr != nullptr;
    // a key tile needs the bias step when there is a bias, or when it is the partial last tile (masking)
    auto uses_slab = [&](const WorkItem &w, int j) { return has_bias || (w.ragged_tail && j == w.n_kv - 1); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 32 * kProducerWarp) {
        // an earlier CTA that gave up leaves the status word raised: later CTAs then skip their work
        sh.abort_flag = (*(volatile unsigned int *)status != 0) ? 1u : 0u;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.q_full[i], 1);
            mbar_init(&sh.q_empty[i], kIssuers);
        }
        for (int i = 0; i < kTiles; ++i) {
            mbar_init(&sh.s_full[i], 1);
            mbar_init(&sh.p_full[i], kBlockM);
            mbar_init(&sh.o_done[i], 1);
        }
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&sh.kv_full[i], 2);   // the TMA loads and the bias slab
            mbar_init(&sh.kv_empty[i], kIssuers);
        }
        mbar_init(&sh.q_slab_full, 1);
        mbar_init(&sh.drained, kIssuers);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kIssuerWarp0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const int height = picked_height(sh, planned, host_plan);
    const int total_items = sh.plan[height - 1].x;
    // All of the SM's tensor memory is allocated, so its base is column 0: the tensor-memory addresses are constants.
    constexpr uint32_t tmem = 0;
    // Register budget: the producer / issuer warpgroup needs few registers and hands its share to the softmax warpgroups
    // (640 x 96 at launch = 61440 = 16 x 32 x 104 + 4 x 32 x 64).  Every warp of a warpgroup executes its setmaxnreg.
    const bool dead = sh.abort_flag != 0 || sh.tmem_base != tmem;  // read after the barrier: uniform for the CTA

    if (dead) {
        if (threadIdx.x == 0 && sh.tmem_base != tmem) atomicOr(status, kErrTmem);
    } else if (warp >= kProducerWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == kProducerWarp) {
            // ===== producer =================================================================================
            const T *bias = reinterpret_cast<const T *>(bias_ptr);
            bool ok = true;
            {   // the constant A side of the bias step: columns 0 and 1 are 1.0.  Both slabs are bfloat16 whatever the
                // q/k/v dtype (the bias step is an MMA instruction of its own): bias/scale and the mask value need its range.
                const uint32_t ones = pack2<true>(1.0f, 1.0f);
                const uint32_t qs = smem_u32(sh.q_slab), ks = smem_u32(sh.k_slab);
                for (int i = lane * 4; i < kQSlabBytes; i += 128) st_shared_u32(qs + i, 0u);
                for (int i = lane * 4; i < kStages * kSlabBytes; i += 128) st_shared_u32(ks + i, 0u);
                __syncwarp();
                for (int i = lane; i < kBlockM; i += 32) st_shared_u32(qs + slab_offset(i), ones);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.q_slab_full);
            }
            int it = 0;      // ring position = key tiles loaded so far
            int q_uses = 0;  // items whose Q was loaded so far (buffer and phase of q_full / q_empty)
            for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
                const WorkItem w = decode_item<kPrefix>(item, sh, work, host_plan, prefix, height);
                if (!w.valid) continue;
                if (lane == 0) {
                    // Item n uses Q buffer n & 1, free once the last tensor-core work of item n - 2 has completed: the next
                    // item's query tiles are in flight while the current item is being computed.
                    const int b = q_uses & 1;
                    if (q_uses >= 2) ok = mbar_wait(&sh.q_empty[b], ((q_uses >> 1) - 1) & 1, sh, status, kErrQFull);
                    if (ok) {
                        mbar_arrive_expect_tx(&sh.q_full[b], w.n_mt * kQTileBytes);
                        for (int t = 0; t < w.n_mt; ++t)
                            tma_load_3d(sh.q[b][w.t0 + t], &map_q, 0, w.head, w.q_row0 - q_begin + t * kBlockM, &sh.q_full[b]);
                    }
                }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                ++q_uses;
                // bias of the lane's keys, fetched one key tile ahead of its use
                float next_bias[kBlockN / 32];
                auto fetch_bias = [&](int j) {
#pragma unroll
                    for (int i = 0; i < kBlockN / 32; ++i) {
                        const int key = w.s0 + j * kBlockN + i * 32 + lane;
                        next_bias[i] = key < w.s1 && has_bias ? Elem<T>::to_f32(bias[key]) : 0.0f;
                    }
                };
                fetch_bias(0);
                for (int j = 0; j < w.n_kv && ok; ++j, ++it) {
                    const int st = it % kStages;
                    if constexpr (kSelfTest) {
                        if (it >= stall_tile) {  // the waits for this tile run out
                            ok = false;
                            break;
                        }
                    }
                    ok = mbar_wait(&sh.kv_empty[st], ((it / kStages) & 1) ^ 1, sh, status, kErrKvEmpty);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_arrive_expect_tx(&sh.kv_full[st], 2 * kKvTileBytes);
                        tma_load_3d(sh.k[st], &map_k, 0, w.head, w.s0 + j * kBlockN, &sh.kv_full[st]);
                        tma_load_3d(sh.v[st], &map_v, 0, w.head, w.s0 + j * kBlockN, &sh.kv_full[st]);
                    }
                    if (uses_slab(w, j)) {
                        const uint32_t ks = smem_u32(sh.k_slab[st]);
#pragma unroll
                        for (int i = 0; i < kBlockN / 32; ++i) {
                            const bool masked = w.s0 + j * kBlockN + i * 32 + lane >= w.s1;
                            const float b = next_bias[i] * inv_scale;
                            const float hi = masked ? kMasked : __bfloat162float(__float2bfloat16_rn(b));
                            st_shared_u32(ks + slab_offset(i * 32 + lane), pack2<true>(hi, masked ? 0.0f : b - hi));
                        }
                        fence_proxy_async();
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.kv_full[st]);
                    if (j + 1 < w.n_kv) fetch_bias(j + 1);
                }
            }
            if (lane == 0) {  // the last use of every buffer has landed before the shared memory is released
                for (int i = max(it - kStages, 0); i < it; ++i)
                    mbar_drain(&sh.kv_full[i % kStages], (i / kStages) & 1, status, kErrKvFull);
                for (int n = max(q_uses - 2, 0); n < q_uses; ++n) mbar_drain(&sh.q_full[n & 1], (n >> 1) & 1, status, kErrQFull);
            }
            __syncwarp();
        } else if (warp < kIssuerWarp0 + kIssuers) {
            // ===== MMA issuers: query tiles first, first + kIssuers, ... ====================================
            // One copy of the code per issuer and uniform control flow, so that the operands of the tensor-core instructions
            // are constants or uniform registers; one elected lane issues a tile's group.
            auto run = [&](auto first_c) {
                constexpr int first = decltype(first_c)::value;
                constexpr uint32_t idesc_qk = make_idesc(kBF16, kBlockM, kBlockN, false);
                constexpr uint32_t idesc_slab = make_idesc(true, kBlockM, kBlockN, false);
                constexpr uint32_t idesc_pv = make_idesc(kBF16, kBlockM, kHeadDim, true);
                const uint64_t q_desc0 = make_smem_desc(smem_u32(sh.q));
                const uint64_t q_slab_desc = make_slab_desc(smem_u32(sh.q_slab), kBlockM);
                const uint64_t k_desc0 = make_smem_desc(smem_u32(sh.k));
                const uint64_t v_desc0 = make_smem_desc(smem_u32(sh.v));
                const uint64_t k_slab_desc0 = make_slab_desc(smem_u32(sh.k_slab), kBlockN);
                // S_t = Q_t K^T (+ the bias step) from ring stage st and Q buffer b
                auto qk = [&](int t, uint32_t st, uint32_t b, bool slab) {
                    const uint32_t s_tmem = tmem + kTmemS + t * kBlockN;
                    const uint64_t qd = q_desc0 + (uint64_t)((b * kTiles + t) * (kQTileBytes >> 4));
                    const uint64_t kd = k_desc0 + (uint64_t)(st * (kKvTileBytes >> 4));
                    tc_mma_ss_1(s_tmem, qd + 0, kd + 0, idesc_qk, 0u);
                    tc_mma_ss_1(s_tmem, qd + 2, kd + 2, idesc_qk, 1u);
                    tc_mma_ss_1(s_tmem, qd + 4, kd + 4, idesc_qk, 1u);
                    tc_mma_ss_1(s_tmem, qd + 6, kd + 6, idesc_qk, 1u);
                    if (slab) tc_mma_ss_1(s_tmem, q_slab_desc, k_slab_desc0 + (uint64_t)(st * (kSlabBytes >> 4)), idesc_slab, 1u);
                    tc_commit_1(&sh.s_full[t]);
                };
                // O_t += P_t V: 16 keys per instruction = 8 columns of 16-bit pairs of P, 16 rows (2048 bytes) of the V tile
                auto pv = [&](int t, uint32_t st, uint32_t accumulate) {
                    const uint32_t o_tmem = tmem + kTmemO + t * kHeadDim, p_tmem = tmem + kTmemS + t * kBlockN;
                    const uint64_t vd = v_desc0 + (uint64_t)(st * (kKvTileBytes >> 4));
#pragma unroll
                    for (int i = 0; i < kBlockN / 16; ++i)
                        tc_mma_ts_1(o_tmem, p_tmem + 8 * i, vd + (uint64_t)(i * 128), idesc_pv, i > 0 ? 1u : accumulate);
                };
                struct Item {
                    uint32_t active;  // bit t: query tile t
                    int n_kv;
                    bool ragged;
                };
                auto next_valid = [&](int &item, Item &x) -> bool {
                    for (; item < total_items; item += gridDim.x) {
                        const WorkItem w = decode_item<kPrefix>(item, sh, work, host_plan, prefix, height);
                        if (w.valid) {
                            x = Item{((1u << w.n_mt) - 1u) << w.t0, w.n_kv, w.ragged_tail};
                            return true;
                        }
                    }
                    return false;
                };
                auto item_slab = [&](const Item &x, int j) { return has_bias || (x.ragged && j == x.n_kv - 1); };
                uint32_t st = 0, kv_phase = 0;  // ring stage of the current key tile; phase of kv_full for the stage after it
                uint32_t p_phase = 0;           // bit t: phase of p_full[t]
                uint32_t qb = 0, q_phase = 0;   // Q buffer of the current item; bit b: phase of q_full[b]
                int item = blockIdx.x;
                Item w, nx;
                bool have = next_valid(item, w);
                // A lane's own "no wait has given up": after a failure its elected lane issues nothing more and its waits try their
                // barrier once.  It does not steer the key loop (that would make the operands non-uniform) except by a vote every
                // 32 key tiles.  A branch on it in front of every wait measured 0.3 % slower.
                bool ok = true;
                auto wait = [&](uint64_t &bar, uint32_t parity, uint32_t code) {
                    if (!mbar_try_wait(&bar, parity)) ok = ok && mbar_wait(&bar, parity, sh, status, code);
                };
                wait(sh.q_slab_full, 0, kErrQFull);
                if (have) {  // the first scores of the first item; later items' first scores are issued with the last P V before them
                    wait(sh.q_full[0], 0, kErrQFull);
                    wait(sh.kv_full[0], 0, kErrKvFull);
                    q_phase ^= 1u;
                    __syncwarp();
                    tc_fence_after();
                    if (elect_one() && ok) {
#pragma unroll
                        for (int t = first; t < kTiles; t += kIssuers)
                            if ((w.active >> t) & 1u) qk(t, 0, 0, item_slab(w, 0));
                        if (w.n_kv == 1) tc_commit_1(&sh.q_empty[0]);
                    }
                    __syncwarp();
                }
                while (have) {
                    // key tiles with a successor in the same item
                    for (int j = 0; j < w.n_kv - 1; ++j) {
                        if ((j & 31) == 31 && !__all_sync(0xffffffffu, ok)) {
                            ok = false;
                            break;
                        }
                        const uint32_t st2 = (st + 1) % kStages;
                        if (st2 == 0) kv_phase ^= 1u;
                        wait(sh.kv_full[st2], kv_phase, kErrKvFull);
                        const bool slab2 = item_slab(w, j + 1);
#pragma unroll
                        for (int t = first; t < kTiles; t += kIssuers) {
                            if ((w.active >> t) & 1u) {
                                // O_t += P_t V, then the next scores of the tile over P_t: the tensor core executes them in order
                                wait(sh.p_full[t], (p_phase >> t) & 1, kErrPFull);
                                p_phase ^= 1u << t;
                                __syncwarp();
                                tc_fence_after();
                                if (elect_one() && ok) {
                                    pv(t, st, j > 0 ? 1u : 0u);
                                    qk(t, st2, qb, slab2);
                                }
                                __syncwarp();
                            }
                        }
                        if (elect_one() && ok) tc_commit_1(&sh.kv_empty[st]);
                        __syncwarp();
                        st = st2;
                    }
                    // last key tile: its scores' successor is the first key tile of the next item, if there is one
                    int item2 = item + gridDim.x;
                    const bool have2 = next_valid(item2, nx);
                    const uint32_t st2 = (st + 1) % kStages;
                    bool slab2 = false;
                    if (st2 == 0) kv_phase ^= 1u;
                    if (!have2) nx.active = 0;
                    else slab2 = item_slab(nx, 0);
                    const uint32_t multi = w.n_kv > 1 ? 1u : 0u;
#pragma unroll
                    for (int t = first; t < kTiles; t += kIssuers) {
                        if ((w.active >> t) & 1u) {
                            wait(sh.p_full[t], (p_phase >> t) & 1, kErrPFull);
                            p_phase ^= 1u << t;
                            __syncwarp();
                            tc_fence_after();
                            if (elect_one() && ok) {
                                pv(t, st, multi);
                                tc_commit_1(&sh.o_done[t]);
                            }
                        }
                        __syncwarp();
                        if (t == first && have2) {  // the next item's first loads: the P V in front needs none of them
                            wait(sh.kv_full[st2], kv_phase, kErrKvFull);
                            wait(sh.q_full[qb ^ 1], (q_phase >> (qb ^ 1)) & 1, kErrQFull);
                            q_phase ^= 1u << (qb ^ 1);
                            __syncwarp();
                        }
                        if (((nx.active >> t) & 1u) && elect_one() && ok) qk(t, st2, qb ^ 1, slab2);
                        __syncwarp();
                    }
                    if (elect_one() && ok) {
                        tc_commit_1(&sh.kv_empty[st]);
                        // Q is free behind the last scores; here with the last P V, except where an item is one key tile
                        if (w.n_kv > 1) tc_commit_1(&sh.q_empty[qb]);
                        if (have2 && nx.n_kv == 1) tc_commit_1(&sh.q_empty[qb ^ 1]);
                    }
                    __syncwarp();
                    st = st2;
                    qb ^= 1u;
                    item = item2;
                    w = nx;
                    have = have2 && __all_sync(0xffffffffu, ok && sh.abort_flag == 0);
                }
                // all tensor-core work and all its commits have arrived before the CTA may end
                __syncwarp();
                if (elect_one()) tc_commit_1(&sh.drained);
                __syncwarp();
                mbar_drain(&sh.drained, 0, status, kErrODone);
                __syncwarp();
            };
            if (warp == kIssuerWarp0) run(std::integral_constant<int, 0>{});
            else run(std::integral_constant<int, 1>{});
        }
    } else {
        // ===== softmax group of query tile t ================================================================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        const int t = warp >> 2;
        const int r = threadIdx.x & 127;                          // row inside the tile == TMEM lane
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t s_tmem = tmem + lane_addr + kTmemS + t * kBlockN;  // P goes over the first half of the scores
        const uint32_t o_tmem = tmem + lane_addr + kTmemO + t * kHeadDim;
        bool ok = true;
        uint32_t s_phase = 0, o_phase = 0;
        struct Item {
            int n_kv, row, q_hi, head, kpart;
        };
        auto next_active = [&](int &item, Item &x) -> bool {
            for (; item < total_items; item += gridDim.x) {
                const WorkItem w = decode_item<kPrefix>(item, sh, work, host_plan, prefix, height);
                if (w.valid && (unsigned)(t - w.t0) < (unsigned)w.n_mt) {
                    x = Item{w.n_kv, w.q_row0 + (t - w.t0) * kBlockM + r, w.q_hi, w.head, w.kpart};
                    return true;
                }
            }
            return false;
        };
        int item = blockIdx.x;
        Item w;
        bool have = next_active(item, w);
        while (have && ok) {
            const int n_kv = w.n_kv;
            float m_ref = -INFINITY, l = 0.0f;  // reference max (log2 units, scale applied) and running sum

            for (int j = 0; j < n_kv; ++j) {
                // The scores of key tile j are complete, and with them (in order) P V of key tile j - 1: the accumulator is
                // stable and P may be overwritten.
                ok = mbar_wait(&sh.s_full[t], s_phase, sh, status, kErrSFull);
                s_phase ^= 1u;
                __syncwarp();
                tc_fence_after();
                constexpr int kHalves = kBlockN / 32;
                uint32_t srow[kHalves][32];
#pragma unroll
                for (int q = 0; q < kHalves; ++q) tmem_ld32(s_tmem + 32 * q, srow[q]);
                tc_wait_ld();
                // Row max over all scores first: independent 3-input chains of 16 scores keep the ALU pipe fed, and the
                // rare rescale is decided once per key tile, so the exponentials below are one straight-line block.
                float t_max = -INFINITY;
#pragma unroll
                for (int c = 0; c < 2 * kHalves; ++c) {
                    const uint32_t *e = &srow[c >> 1][(c & 1) * 16];
                    float m = max3(__uint_as_float(e[0]), __uint_as_float(e[1]), __uint_as_float(e[2]));
#pragma unroll
                    for (int i = 3; i < 15; i += 2) m = max3(m, __uint_as_float(e[i]), __uint_as_float(e[i + 1]));
                    t_max = max3(t_max, m, __uint_as_float(e[15]));
                }
                t_max *= scale_log2;
                const bool need = t_max > m_ref + kRescaleThreshold;  // always true on the first key tile (m_ref = -inf)
                if (__any_sync(0xffffffffu, need || !ok)) {
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    float alpha = 1.0f;
                    if (need) {
                        alpha = (m_ref == -INFINITY) ? 0.0f : fast_exp2(m_ref - t_max);
                        m_ref = t_max;
                        l *= alpha;
                    }
                    if (j > 0) scale_accumulator(o_tmem, alpha);  // rescale what earlier key tiles accumulated
                }
                // p = 2^(s * scale*log2e - m_ref), two scores per instruction; a share of the pairs takes the polynomial
                // route so that the special-function unit and the FMA pipe split the exponentials.
                const f32x2_t scale2 = pack_f32x2(scale_log2, scale_log2), neg_m2 = pack_f32x2(-m_ref, -m_ref);
                f32x2_t sum2 = pack_f32x2(0.0f, 0.0f);
#pragma unroll
                for (int q = 0; q < kHalves; ++q) {
                    uint32_t pk[16];
#pragma unroll
                    for (int pair = 0; pair < 16; ++pair) {
                        const f32x2_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(srow[q][2 * pair]), __uint_as_float(srow[q][2 * pair + 1])), scale2, neg_m2);
                        float x0, x1, p0, p1;
                        unpack_f32x2(x2, x0, x1);
                        if ((kPolyPairs >> pair) & 1u) {
                            exp2_poly_x2(x0, x1, p0, p1);
                        } else {
                            p0 = fast_exp2(x0);
                            p1 = fast_exp2(x1);
                        }
                        sum2 = add_f32x2(sum2, pack_f32x2(p0, p1));
                        pk[pair] = pack2<kBF16>(p0, p1);
                    }
                    tmem_st16(s_tmem + 16 * q, pk);  // 32 keys -> 16 columns of 16-bit pairs
                }
                {
                    float s_lo, s_hi;
                    unpack_f32x2(sum2, s_lo, s_hi);
                    l += s_lo + s_hi;
                }
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(&sh.p_full[t]);
            }

            // While the last P V runs: the next item, and what this one's epilogue needs beside the accumulator.
            const bool in_range = w.row < w.q_hi;
            const int64_t row = w.row - q_begin;
            T *dst_row = reinterpret_cast<T *>(out_ptr) + (int64_t)w.kpart * part_o + row * o_rs + (int64_t)w.head * kHeadDim;
            float *dst_lse = lse + (int64_t)w.kpart * part_l + (int64_t)w.head * (q_end - q_begin) + row;
            item += gridDim.x;
            have = next_active(item, w);
            const float inv = 1.0f / l, row_lse = (m_ref + log2f(l)) * kLn2;
            if (ok) {
                ok = mbar_wait(&sh.o_done[t], o_phase, sh, status, kErrODone);
                o_phase ^= 1u;
                ok = __all_sync(0xffffffffu, ok);
            }
            if (ok) {
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t o[32], pk[16];
                    tmem_ld32(o_tmem + 32 * c, o);
                    tc_wait_ld();  // the next item's first P V, which overwrites the accumulator, waits for this group's next P
                    if (in_range) {
                        // The row's outputs as packed words, written with 32-byte stores where the address allows it: a warp's
                        // store then covers whole 32-byte sectors of its 32 rows instead of halves.
#pragma unroll
                        for (int i = 0; i < 32; i += 2)
                            pk[i / 2] = pack2<kBF16>(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                        if ((reinterpret_cast<uintptr_t>(dst_row) & 31) == 0) {
#pragma unroll
                            for (int i = 0; i < 16; i += 8)
                                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst_row + 32 * c + 2 * i),
                                             "r"(pk[i]), "r"(pk[i + 1]), "r"(pk[i + 2]), "r"(pk[i + 3]), "r"(pk[i + 4]), "r"(pk[i + 5]),
                                             "r"(pk[i + 6]), "r"(pk[i + 7])
                                             : "memory");
                        } else {
                            uint4 *dst = reinterpret_cast<uint4 *>(dst_row + 32 * c);
#pragma unroll
                            for (int i = 0; i < 16; i += 4) dst[i / 4] = make_uint4(pk[i], pk[i + 1], pk[i + 2], pk[i + 3]);
                        }
                    }
                    __syncwarp();
                }
                if (lse && in_range) *dst_lse = row_lse;
                tc_fence_before();  // the accumulator has been read; ordered before the next arrival on p_full
            }
        }
    }
    // ===== common exit ==========================================================================================
    tc_fence_before();
    __syncthreads();
    if (warp == kIssuerWarp0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem_base), "r"(kTmemCols) : "memory");
    }
}

// Self-test of the failure path: one CTA waits, with the attention kernel's own bounded wait, on a barrier that nothing
// ever arrives at.  The wait gives up after `ticks` clocks, raises the CTA's abort flag and the device status word, and
// the kernel returns normally; `waited_out` (optional) receives the clocks it waited.
__global__ void selftest_wait_kernel(long long ticks, unsigned int *__restrict__ status, long long *__restrict__ waited_out) {
    __shared__ alignas(8) uint64_t bar;
    __shared__ uint32_t abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const long long t0 = clock64();
    const bool ok = mbar_wait_limit(&bar, 0, &abort_flag, status, kErrSelfTest, ticks);
    if (threadIdx.x == 0 && waited_out) *waited_out = ok ? -1 : clock64() - t0;
}

// The work list of a launch on `ctas` CTAs as the attention kernel walks it, for tests: out[0 .. 4) = items, query tiles per
// item, first split item, parts of a split one; then per item head, first and last + 1 key, first query row, end of the query
// rows, query tiles (0: skipped), key tiles, first tile slot.
template <bool kPrefix>
__global__ void __launch_bounds__(kThreads, 1)
work_list_kernel(const int *__restrict__ cu, int q_begin, int q_end, int max_rows, int nseg, int num_heads, const int *__restrict__ max_len_dev, int ctas,
                 const WorkPlan host_plan, int *__restrict__ out, int capacity) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    SharedStorage &sh = *reinterpret_cast<SharedStorage *>(smem_raw);
    WorkArgs work{cu, nseg, num_heads, q_begin, q_end, 0, max_rows, 1, ctas, false};
    if (max_len_dev != nullptr) work.max_rows = min(max_rows, max(*max_len_dev, 0));
    int *prefix = reinterpret_cast<int *>(reinterpret_cast<uint8_t *>(&sh) + sizeof(SharedStorage));
    const int planned = plan_work<kPrefix>(sh, work, host_plan, prefix);
    __syncthreads();
    const int height = picked_height(sh, planned, host_plan);
    const int4 pl = sh.plan[height - 1];
    if (threadIdx.x >= 32) return;
    if (threadIdx.x == 0) {
        out[0] = pl.x;
        out[1] = height;
        out[2] = pl.y;
        out[3] = pl.z;
    }
    for (int item = 0; item < min(pl.x, capacity); ++item) {
        const WorkItem w = decode_item<kPrefix>(item, sh, work, host_plan, prefix, height);
        if (threadIdx.x == 0) {
            int *o = out + 4 + 8 * (int64_t)item;
            o[0] = w.head;
            o[1] = w.s0;
            o[2] = w.s1;
            o[3] = w.q_row0;
            o[4] = w.q_hi;
            o[5] = w.valid ? w.n_mt : 0;
            o[6] = w.n_kv;
            o[7] = w.t0;
        }
    }
}

// ---- host side --------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

// [total, H, 64] view with arbitrary row stride; box = box_rows rows x 1 head x 64 elements, 128-byte swizzle.
// A tensor map is a pure function of these arguments (it holds an address, not a snapshot of memory), so each host
// thread keeps the last few it encoded: a model that calls attention layer after layer on the same buffers encodes
// them once instead of three times per launch.
struct MapKey {
    const void *base;
    int64_t total, row_stride;
    int dtype, H, box_rows;
    bool operator==(const MapKey &o) const {
        return base == o.base && total == o.total && row_stride == o.row_stride && dtype == o.dtype && H == o.H && box_rows == o.box_rows;
    }
};
constexpr int kMapCacheSlots = 16;
struct MapCache {
    MapKey key[kMapCacheSlots];
    CUtensorMap map[kMapCacheSlots];
    bool used[kMapCacheSlots];
    int next;
};

int make_map(CUtensorMap *map, const void *base, int dtype, int64_t total, int H, int64_t row_stride, int box_rows) {
    thread_local MapCache cache = {};
    const MapKey key{base, total, row_stride, dtype, H, box_rows};
    for (int i = 0; i < kMapCacheSlots; ++i)
        if (cache.used[i] && cache.key[i] == key) {
            *map = cache.map[i];
            return COME_OK;
        }
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the CUDA driver");
        return COME_ERR_CUDA;
    }
    cuuint64_t dims[3] = {(cuuint64_t)kHeadDim, (cuuint64_t)H, (cuuint64_t)total};
    cuuint64_t strides[2] = {(cuuint64_t)kHeadDim * 2, (cuuint64_t)row_stride * 2};
    cuuint32_t box[3] = {(cuuint32_t)kHeadDim, 1, (cuuint32_t)box_rows};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, dtype == COME_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                    const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return COME_ERR_CUDA;
    }
    const int slot = cache.next;
    cache.next = (slot + 1) % kMapCacheSlots;
    cache.key[slot] = key;
    cache.map[slot] = *map;
    cache.used[slot] = true;
    return COME_OK;
}

}  // namespace

bool attn_sm100_supported(const AttnArgs &a) {
    if (a.D != kHeadDim) return false;
    if (a.dtype != COME_BF16 && a.dtype != COME_F16) return false;
    auto al16 = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
    if (!al16(a.q) || !al16(a.k) || !al16(a.v) || !al16(a.out)) return false;
    if (a.q_rs % 8 || a.k_rs % 8 || a.v_rs % 8 || a.o_rs % 8) return false;
    // the row max is taken on raw scores and the bias is divided by the scale: both need a positive finite scale
    if (!(a.scale > 0.0f) || !(a.scale < 3.0e38f)) return false;
    return true;
}

// The shared-memory opt-in of a kernel is set once per device and instantiation (not again on every launch, so that
// launches stay cheap and legal inside a stream capture).  Host threads may race to the first launch: the flag is
// raised only after cudaFuncSetAttribute has succeeded, under a mutex, so no thread launches before the opt-in exists
// and a failed attempt is retried by the next launch.
template <typename Kernel> static int ensure_smem_optin(Kernel kernel, int slot, size_t smem) {
    static std::mutex mu;
    static bool done[64][7];
    int dev = 0;
    COME_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("come_attn_varlen_fwd: device ordinal %d is out of the supported range", dev);
        return COME_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev][slot]) return COME_OK;
    COME_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    done[dev][slot] = true;
    return COME_OK;
}

// Upper bound on the CTAs of the persistent kernel for launches issued by this host thread (0 = one per SM).
static thread_local int t_cta_limit = 0;
void attn_sm100_set_cta_limit(int max_ctas) { t_cta_limit = max_ctas > 0 ? max_ctas : 0; }

struct LaunchPlan {
    WorkPlan work;
    bool with_table;
    int span;       // most query rows a segment can own in this launch
    unsigned grid;
    int64_t items;  // upper bound; nothing to launch when it is 0
};

static int plan_launch(const AttnArgs &a, LaunchPlan *out) {
    const int64_t q_rows = a.q_end - a.q_begin;
    const int64_t span = a.q_free ? q_rows : (a.max_seqlen < q_rows ? a.max_seqlen : q_rows);  // most query rows any segment can own here
    int sms = sm_count();
    if (t_cta_limit > 0 && t_cta_limit < sms) sms = t_cta_limit;
    // Query tiles per work item: chosen on the device from the segments (0) where there are several; on the host for one, for
    // launches that give every query tile a CTA, where the caller plans launches by their items (q_free: three tiles, see
    // plan_tail_split) and where a launch has more segments than the table holds.
    const int64_t most_tiles = (span + kBlockM - 1) / kBlockM;  // of one segment
    const bool with_table = !a.q_free && most_tiles > 1 && a.nseg >= kMinPrefixSegs && a.nseg <= kMaxPrefixSegs;
    WorkPlan plan = {};
    if (a.q_free) plan.height = 3;
    else if (most_tiles == 1 || (!with_table && most_tiles * a.nseg * a.H <= sms)) plan.height = 1;
    else if (a.nseg > kMaxPrefixSegs) plan.height = kTiles;
    const bool one_segment = plan.height == 0 && a.nseg == 1 && a.max_seqlen_dev == nullptr;
    const int height = plan.height == 0 ? 1 : plan.height;  // of the lowest items the launch may have
    const int64_t nblk_x = (span + height * kBlockM - 1) / (height * kBlockM);
    const int k_parts = a.k_parts > 1 ? a.k_parts : 1;
    if (k_parts > 1) {
        // shares of the key tiles of every item: one segment whose keys all query rows attend to; no share may be empty
        const int64_t tiles = (a.total + kBlockN - 1) / kBlockN, per_part = (tiles + k_parts - 1) / k_parts;
        if (!a.q_free || a.lse == nullptr || (int64_t)(k_parts - 1) * per_part >= tiles) {
            set_error("attention with %d key shares needs the one-segment cross form, a log-sum-exp output and at least one "
                      "key tile per share (%lld tiles)", k_parts, (long long)tiles);
            return COME_ERR_ARG;
        }
    }
    // an exact list holds no more than the rows' tiles and a partial one per segment, however loose max_seqlen is
    const int64_t slots = nblk_x * a.nseg, blocks = plan.height == 0 ? std::min(slots, q_rows / kBlockM + a.nseg) : slots;
    const int64_t items = blocks * a.H * k_parts, slot_items = slots * a.H * k_parts;
    out->items = items;
    out->span = (int)span;
    out->with_table = with_table;
    if (items <= 0) return COME_OK;
    if (items >= (1ll << 31)) {
        set_error("come_attn_varlen_fwd: %lld work items do not fit 32 bits", (long long)items);
        return COME_ERR_ARG;
    }
    const unsigned grid = out->grid = (unsigned)(slot_items < sms ? slot_items : sms);  // persistent: one CTA per SM walks the items
    if (one_segment) {
        const int n = (int)most_tiles;
        float least = 3.0e38f;
        for (int h = kTiles; h >= 1; --h) {
            WorkPlan p = {};
            const int blocks = blocks_of(n, h), total = blocks * a.H, rest = total % (int)grid, rounds = total / (int)grid + (rest > 0 ? 1 : 0);
            const float mean = (float)height_cost(n, h) / (float)blocks;
            const float cost = split_last_round(p, h, total, rest, (float)rounds * mean, mean, 1.0f, (int)grid);
            if (cost < least) {
                least = cost;
                plan = p;
                plan.slots = blocks;
            }
        }
    } else if (plan.height != 0) {
        plan.slots = (int)nblk_x;
        plan.total = plan.from = (int)items;
        plan.parts = 1;
    }
    auto reciprocal = [](int64_t d) { return d > 0 ? (uint32_t)(0xffffffffu / (uint64_t)d) : 0u; };
    plan.slots_rcp = reciprocal(plan.slots);
    plan.nseg_rcp = reciprocal(a.nseg);
    plan.ctas_rcp = reciprocal(grid);
    out->work = plan;
    return COME_OK;
}

int attn_sm100_launch(const AttnArgs &a, cudaStream_t stream) {
    unsigned int *status = status_word_dev();
    if (!status) return COME_ERR_CUDA;
    CUtensorMap mq, mk, mv;
    int rc;
    if ((rc = make_map(&mq, a.q, a.dtype, a.q_end - a.q_begin, a.H, a.q_rs, kBlockM)) != COME_OK) return rc;
    if ((rc = make_map(&mk, a.k, a.dtype, a.total, a.H, a.k_rs, kBlockN)) != COME_OK) return rc;
    if ((rc = make_map(&mv, a.v, a.dtype, a.total, a.H, a.v_rs, kBlockN)) != COME_OK) return rc;
    LaunchPlan plan;
    if ((rc = plan_launch(a, &plan)) != COME_OK) return rc;
    if (plan.items <= 0) return COME_OK;
    const bool with_table = plan.with_table;
    const unsigned grid = plan.grid;
    const size_t smem = sizeof(SharedStorage) + 1024 + (with_table ? kPrefixTableBytes : 0);
    const int k_parts = a.k_parts > 1 ? a.k_parts : 1;
    const float scale_log2 = a.scale * kLog2e;
    const float inv_scale = 1.0f / a.scale;
#define COME_ATTN_LAUNCH(BF16, PREFIX, SELFTEST, SLOT)                                                                         \
    do {                                                                                                                       \
        if ((rc = ensure_smem_optin(attn_fwd_sm100_kernel<BF16, PREFIX, SELFTEST>, SLOT, smem)) != COME_OK) return rc;          \
        attn_fwd_sm100_kernel<BF16, PREFIX, SELFTEST><<<grid, kThreads, smem, stream>>>(mq, mk, mv, a.bias, a.cu, scale_log2, inv_scale, a.out, \
                                                                              a.o_rs, a.lse, (int)a.q_begin, (int)a.q_end, plan.span, \
                                                                              a.nseg, a.H, a.max_seqlen_dev, status, (int)a.total,   \
                                                                              a.q_free ? 1 : 0, k_parts, (long long)a.part_o, \
                                                                              (long long)a.part_l, plan.work, a.stall_tile);         \
    } while (0)
    if (a.stall_tile >= 0) {
        COME_ATTN_LAUNCH(true, false, true, 4);
    } else if (a.dtype == COME_BF16) {
        if (with_table) COME_ATTN_LAUNCH(true, true, false, 0);
        else COME_ATTN_LAUNCH(true, false, false, 1);
    } else {
        if (with_table) COME_ATTN_LAUNCH(false, true, false, 2);
        else COME_ATTN_LAUNCH(false, false, false, 3);
    }
#undef COME_ATTN_LAUNCH
    return check_launch("come_attn_varlen_fwd (tcgen05 kernel)");
}

}  // namespace come

extern "C" int come_selftest_bounded_wait(int64_t ticks, int64_t *waited_dev, void *stream) {
    COME_REQUIRE(ticks > 0 && ticks <= (1ll << 26), "come_selftest_bounded_wait: ticks must be in (0, 2^26] (a fraction of a second)");
    unsigned int *status = come::status_word_dev();
    if (!status) return COME_ERR_CUDA;
    come::selftest_wait_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((long long)ticks, status, (long long *)waited_dev);
    return come::check_launch("come_selftest_bounded_wait");
}

extern "C" int come_selftest_attn_stall(const void *qkv_dev, int64_t total, int num_heads, const int32_t *cu_seqlens_dev, float softmax_scale,
                                        int key_tiles, void *out_dev, float *lse_dev, void *stream) {
    COME_REQUIRE(qkv_dev && cu_seqlens_dev && out_dev, "come_selftest_attn_stall: qkv, cu_seqlens and out must be given");
    COME_REQUIRE(total > 0 && total < (1ll << 20) && num_heads > 0 && num_heads <= 64, "come_selftest_attn_stall: a small launch only (tokens below 2^20, at most 64 heads)");
    COME_REQUIRE(key_tiles >= 0, "come_selftest_attn_stall: key_tiles must not be negative");
    come::AttnArgs a = {};
    const int64_t part = (int64_t)num_heads * come::kHeadDim;  // elements of q, of k and of v in a packed row
    const uint16_t *qkv = static_cast<const uint16_t *>(qkv_dev);
    a.q = qkv;
    a.k = qkv + part;
    a.v = qkv + 2 * part;
    a.cu = cu_seqlens_dev;
    a.out = out_dev;
    a.lse = lse_dev;
    a.dtype = COME_BF16;
    a.total = a.q_end = total;
    a.H = num_heads;
    a.D = come::kHeadDim;
    a.q_rs = a.k_rs = a.v_rs = 3 * part;
    a.o_rs = part;
    a.nseg = 1;
    a.max_seqlen = (int)total;
    a.scale = softmax_scale;
    a.k_parts = 1;
    a.stall_tile = key_tiles;
    COME_REQUIRE(come::attn_sm100_supported(a), "come_selftest_attn_stall: needs 16-byte aligned tensors and a positive scale");
    return come::attn_sm100_launch(a, (cudaStream_t)stream);
}

extern "C" int come_attn_work_list(const int32_t *cu_seqlens_dev, int num_segments, int num_heads, int64_t q_row_begin, int64_t q_row_end,
                                   int max_seqlen, const int32_t *max_seqlen_dev, int max_ctas, int32_t *out_dev, int64_t capacity, void *stream) {
    COME_REQUIRE(cu_seqlens_dev && out_dev && num_segments > 0 && num_heads > 0 && max_seqlen > 0 && capacity >= 0 && capacity < (1ll << 28),
                 "come_attn_work_list: bad arguments");
    COME_REQUIRE(q_row_begin >= 0 && q_row_begin < q_row_end && q_row_end < (1ll << 31), "come_attn_work_list: bad row range");
    using namespace come;
    AttnArgs a = {};
    a.q_begin = q_row_begin;
    a.q_end = q_row_end;
    a.H = num_heads;
    a.nseg = num_segments;
    a.max_seqlen = max_seqlen;
    a.max_seqlen_dev = max_seqlen_dev;
    LaunchPlan plan;
    const int limit = t_cta_limit;
    t_cta_limit = max_ctas;
    int rc = plan_launch(a, &plan);
    t_cta_limit = limit;
    if (rc != COME_OK) return rc;
    const size_t smem = sizeof(SharedStorage) + 1024 + kPrefixTableBytes;
    if (plan.with_table) {
        if ((rc = ensure_smem_optin(work_list_kernel<true>, 5, smem)) != COME_OK) return rc;
        work_list_kernel<true><<<1, kThreads, smem, (cudaStream_t)stream>>>(cu_seqlens_dev, (int)q_row_begin, (int)q_row_end, plan.span, num_segments, num_heads,
                                                                            max_seqlen_dev, (int)plan.grid, plan.work, out_dev, (int)capacity);
    } else {
        if ((rc = ensure_smem_optin(work_list_kernel<false>, 6, smem)) != COME_OK) return rc;
        work_list_kernel<false><<<1, kThreads, smem, (cudaStream_t)stream>>>(cu_seqlens_dev, (int)q_row_begin, (int)q_row_end, plan.span, num_segments, num_heads,
                                                                             max_seqlen_dev, (int)plan.grid, plan.work, out_dev, (int)capacity);
    }
    return check_launch("come_attn_work_list");
}
