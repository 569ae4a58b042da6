// The dense layers on the 5th-generation tensor cores: tcgen05.mma (kind::f16, bf16 operands) with FP32 accumulation in
// tensor memory.  Every operand is split into three bf16 numbers, and six of the nine products are formed:
//
//   x = x0 + x1 + x2 (8 significant bits each; exact for |x| above 2^-110, below which x2 falls under bf16's smallest number)
//   A B^T  ~  A0 B0^T + (A0 B1^T + A1 B0^T + A1 B1^T + A0 B2^T + A2 B0^T)      (what is dropped is below 2^-24 of a product)
//
// at the price of three TF32 products, whose two parts lose two bits of an operand.
// Accuracy: the tensor core cuts off what does not fit when it adds to its accumulator, so one accumulator for everything
// would collect an error of one sign per instruction.  The A0 B0 products therefore go in turns to three accumulators and
// the small products to a fourth; the epilogue adds the four in FP32.  Distance from 64 bits, of the result's norm, for
// normal operands and 128 / 512 terms: 6.6e-8 / 7.8e-8 (16e-8 where one block takes all 512); a chain of FP32 fused
// multiply-adds 20e-8 / 21e-8 (41e-8), three TF32 products 16e-8 / 16e-8 (44e-8).  Operands of one sign: 7.1e-8 / 6.9e-8
// (22e-8) against 17e-8 / 9.5e-8 (35e-8); ReLU outputs 5.4e-8 / 6.7e-8 (11e-8) against 14e-8 / 15e-8 (29e-8).
// What is cut off grows with the terms, where a chain's error grows with their root, and most for operands of one sign, of
// which nothing averages out.  Longer contractions therefore go in runs: the A0 B0 products to two accumulators, which
// together with the small ones are added in FP32, behind every run, to a sum in the third one's place (tc_drain).
// Products of more than 512 terms in runs of eight slices, K = 2 048 / 32 768, 1 024 rows, operands of one sign: 17e-8 / 18e-8,
// without runs 22e-8 / 773e-8, FP32 18e-8 / 70e-8; 18 / 220 us, without 17 / 198, FP32 36 / 515.  Weight gradients of splits
// of more than 160 rows in runs of four slices, 4 000 / 10 700 / 131 072 atoms, operands of one sign: 8.4e-8 / 8.2e-8 / 8.8e-8,
// without runs 10e-8 / 26e-8 / 651e-8, FP32 8.5e-8 / 10.9e-8 / 33e-8; of both 10e-8 / 11e-8 / 18e-8, without 11e-8 / 15e-8 /
// 206e-8, FP32 22e-8 / 34e-8 / 118e-8.  Per launch of a layer's two, 2 661 atoms 12.7 us, without runs 11.9; 10 700 33.5 / 30.7.
//
// One CTA of eight warps and one owns a 128 x 64 output tile (or, over a cluster, a part of its contraction).  Per 32-wide slice
// of the contraction index the eight warps bring both operands from global memory through registers (two register sets:
// a slice's loads are in flight behind the one in work), split them, and store the three parts to one of three
// shared-memory stages as they lie in global memory, in the layout the tensor core reads: operands whose contraction index
// is contiguous K-major with 64-byte swizzle (8-row groups of 512 bytes, the 16-byte chunk j of row r stored at chunk
// j ^ ((r >> 1) & 3)), the others (the weight in a data gradient, both operands of a weight gradient) MN-major with 128-byte
// swizzle (blocks of 64 rows; a contraction index is 128 bytes, its chunk j stored at chunk j ^ (k & 7)).  A thread of the
// ninth warp waits for the stage to be full (an mbarrier that each warp arrives at), issues 2 (k-steps of 16) x 6 (products)
// tcgen05.mma instructions and commits them to the stage's other mbarrier, which is waited on before the stage is written
// again three slices later: nobody else waits for the tensor core, whose queue holds up the thread that fills it.  The
// epilogue adds the accumulators (tcgen05.ld; a warp reads the TMEM lanes of its quarter: rows; warps w and w + 4 take half
// of the columns each), leaves the tile in shared memory, and finishes it row by row: bias, residual, ReLU, ReLU mask.
//
// Two CTAs fit an SM (109 KB of shared memory, half of the tensor memory, 96 registers a thread): one splits while the
// other multiplies.  Every kernel here that allocates tensor memory needs as much, so an allocation never waits.
// What bounds it: up to 2 700 rows a chain of latencies (launch, first loads, four slices, epilogue), beyond that the
// instructions of the split (issue slots 48 % busy, tensor pipe 18 %).  Kernel time, [128] -> [512] and [512] -> [128],
// against FP32 in gemm_kernel: 400 rows 7.5 / 8.9 against 7.1 / 8.6 us, 600 rows 7.6 / 9.0 against 10.3 / 11.9, 2 661 rows
// 10.6 / 12.0 against 17.4 / 19.3, 10 700 rows 25 / 25 against 52 / 59; weight gradients of a layer of 10 700 atoms 67 against
// 190.  Measured and left: 16 warps that bring and split, and a block barrier per slice with the instructions issued by one
// of them (27 / 29 us); operands transposed on their way to shared memory (27 / 35 us in data gradients).
//
// Every wait on an mbarrier is bounded: on expiry the kernel sets CFB200_ST_TC_TIMEOUT, goes on with wrong numbers and
// ends.  An operand that is not finite has no split (inf - inf); a tile with a result that is not finite is computed again
// in plain FP32.
//
// No TMA: the operands need the split on the way to shared memory, so they pass through registers anyway.
#include <atomic>
#include <cuda_bf16.h>
#include "common.cuh"

namespace cfb {

constexpr int kTcThreads = 256;              // that bring and split operands, and finish the tile
constexpr int kTcBlock = kTcThreads + 32;    // and the warp that issues the tensor core's instructions
constexpr int kTcM = 128, kTcN = 64;         // rows of the operands per tile
constexpr int kTcKc = 32;                    // contraction slice: 32 bf16 = one 64-byte swizzle row
constexpr int kTcABytes = kTcM * kTcKc * 2, kTcBBytes = kTcN * kTcKc * 2;       // one part: 8 KB, 4 KB
constexpr int kTcStageBytes = 3 * (kTcABytes + kTcBBytes);      // A0, A1, A2, B0, B1, B2
constexpr int kTcStages = 3;
constexpr int kTcSmemBytes = kTcStages * kTcStageBytes + 1024;  // and alignment slack
constexpr int kTcAcc = 3;                    // accumulators of the large products (two, and the sum so far, where there are
                                             // several runs); the small ones' follows them
constexpr int kTcCols = 256;                 // tensor-memory columns: four accumulators
constexpr int kTcTileLd = kTcN / 4 + 1;      // float4 per row of the finished tile (conflict-free writes by rows)
static_assert((kTcM * kTcTileLd + kTcThreads) * 16 <= kTcStages * kTcStageBytes, "the finished tile, and column sums, fit the stages");
// Slices of a contraction that is taken in one run, and of a run (see above): in one run as long as that is no farther from 64
// bits than the chain of FP32 additions in the kernels of the FP32 pipe.
constexpr int kTcWholeGemm = 16, kTcRunGemm = 8, kTcWholeWgrad = 5, kTcRunWgrad = 4;
constexpr uint32_t kTcSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Two numbers into three bf16 each (packed: x low, y high); every step is exact (see above).  A number that is not finite, or rounds to
// infinity, leaves a part that is not a number.
__device__ __forceinline__ void tc_split2(float x, float y, uint32_t (&part)[3])
{
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
        part[i] = *reinterpret_cast<const uint32_t*>(&b);
        if (i < 2) { x -= __uint_as_float(part[i] << 16); y -= __uint_as_float(part[i] & 0xFFFF0000u); }
    }
}

// Shared-memory matrix descriptor, version 1.  K-major, SWIZZLE_64B: 8-row groups 512 bytes apart.  MN-major (TR),
// SWIZZLE_128B: blocks of 64 rows kTcKc x 128 bytes apart, 8 contraction indices 1024 bytes apart.
template <bool TR>
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t saddr)
{
    const uint64_t base = (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)1 << 46);
    if (TR) return base | ((uint64_t)(kTcKc * 128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)2 << 61);
    return base | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)4 << 61);
}

// from one k-step of 16 to the next, in descriptor units of 16 bytes
__host__ __device__ constexpr uint64_t tc_kstep(bool TR) { return TR ? 2 * 1024 >> 4 : 32 >> 4; }

// instruction descriptor: D = F32, A = B = BF16, M = 128, N = 64; bits 15, 16: A, B MN-major
template <bool TRA, bool TRB>
__device__ __forceinline__ constexpr uint32_t tc_idesc()
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((TRA ? 1u : 0u) << 15) | ((TRB ? 1u : 0u) << 16) | ((uint32_t)(kTcN >> 3) << 17) |
           ((uint32_t)(kTcM >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity)
{
    for (uint32_t it = 0; it < kTcSpinLimit; it++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// registers holding one slice of both operands
__host__ __device__ constexpr int tc_float4(int rows) { return rows * kTcKc / 4 / kTcThreads; }
struct TcSlice { float4 a[tc_float4(kTcM)], b[tc_float4(kTcN)]; };

// One operand of a product as one thread fetches it.  Element (r, k) of the operand is src[r * ld + k] (k contiguous) or,
// transposed, src[k * ld + r].  The thread's float4 i of a slice is number tid + 256 i, eight to a row of K or,
// transposed, ROWS / 4 to a contraction index: from one to the next are 32 rows, or 1024 / ROWS indices.
template <int ROWS, bool TR>
struct TcFetch {
    static constexpr int kSkip = TR ? kTcThreads * 4 / ROWS : kTcThreads / 8;    // rows or indices from one float4 to the next
    const float* p;                          // the thread's first float4 of the slice to fetch next
    int step, stride;                        // to the next slice, to the next float4
    int left;                                // rows (transposed: contraction indices) from the thread's first on
    __device__ __forceinline__ static int row() { return TR ? 4 * ((int)threadIdx.x % (ROWS / 4)) : (int)threadIdx.x >> 3; }
    __device__ __forceinline__ static int idx() { return TR ? (int)threadIdx.x / (ROWS / 4) : 4 * ((int)threadIdx.x & 7); }
    // operand rows r0 .. and contraction indices k0 .. on; rows: of the operand.  Transposed: all of its rows exist, and
    // contraction indices up to K do; else all indices of a slice exist
    __device__ __forceinline__ void open(const float* src, const int ld, const int r0, const int rows, const int k0, const int K)
    {
        const size_t r = r0 + row(), k = k0 + idx();
        p = src + (TR ? k * ld + r : r * ld + k);
        step = TR ? kTcKc * ld : kTcKc;
        stride = kSkip * ld;
        left = TR ? K - (int)k : rows - (int)r;
    }
    __device__ __forceinline__ void next(float4* v)
    {
#pragma unroll
        for (int i = 0; i < tc_float4(ROWS); i++) {
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i * kSkip < left) v[i] = __ldg(reinterpret_cast<const float4*>(p + (ptrdiff_t)i * stride));
        }
        p += step;
        if (TR) left -= kTcKc;
    }
    // where the thread's first float4 goes in a part of a stage (half of a 16-byte chunk), and how far the next ones are
    __device__ __forceinline__ static int place()
    {
        const int r = row(), k = idx();
        return TR ? (r >> 6) * (kTcKc * 128) + k * 128 + ((((r >> 3) ^ k) & 7) << 4) + 2 * (r & 4)
                  : r * 64 + (((k >> 3) ^ (r >> 1)) & 3) * 16 + 2 * (k & 4);
    }
    static constexpr int kNext = kSkip * (TR ? 128 : 64);
    static_assert(kSkip % 8 == 0, "the swizzle of a thread's float4 is the same");
};

// splits a slice into its stage, from the thread's place on (the parts of an operand are ROWS * 64 bytes apart)
template <int ROWS, bool TR>
__device__ __forceinline__ void tc_stash1(const float4* v, uint8_t* o)
{
#pragma unroll
    for (int i = 0; i < tc_float4(ROWS); i++) {
        uint32_t lo[3], hi[3];
        tc_split2(v[i].x, v[i].y, lo);
        tc_split2(v[i].z, v[i].w, hi);
#pragma unroll
        for (int p = 0; p < 3; p++)
            *reinterpret_cast<uint2*>(o + i * TcFetch<ROWS, TR>::kNext + p * ROWS * 64) = make_uint2(lo[p], hi[p]);
    }
}

// CTA-wide state of one tile computation: the shared-memory stages with their mbarriers
struct TcCta {
    uint8_t* stage;
    uint32_t full, empty, drained, tmem;     // mbarriers per stage: written by all warps; read by its instructions; of a run:
    uint32_t slices_done;                    // added to the sum so far
    uint32_t runs_drained;
    bool failed;
};
constexpr int kTcBarriers = 2 * kTcStages + 1;

__device__ __forceinline__ void tc_begin(TcCta& T, uint8_t* smem_raw, uint64_t* mbar_slots, uint32_t* tmem_slot)
{
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    T.stage = smem_raw + (base - smem_u32(smem_raw));
    T.full = smem_u32(mbar_slots);
    T.empty = T.full + 8 * kTcStages;
    T.drained = T.empty + 8 * kTcStages;
    T.slices_done = T.runs_drained = 0;
    T.failed = false;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kTcStages; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(T.full + 8 * i), "r"(kTcThreads / 32) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(T.empty + 8 * i) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(T.drained), "r"(kTcThreads / 32) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if ((threadIdx.x >> 5) == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)kTcCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    T.tmem = *tmem_slot;
}

// Splits one 32-wide slice held in registers into the stage slices_done % 3 of shared memory, once the instructions that
// read that stage three slices ago have finished.
template <bool TRA, bool TRB>
__device__ __forceinline__ void tc_slice(TcCta& T, const TcSlice& S)
{
    const uint32_t s = T.slices_done++, round = s / kTcStages, st = s - round * kTcStages;
    if (round > 0 && !tc_wait(T.empty + 8 * st, (round - 1) & 1)) T.failed = true;
    uint8_t* base = T.stage + st * kTcStageBytes;
    tc_stash1<kTcM, TRA>(S.a, base + TcFetch<kTcM, TRA>::place());
    tc_stash1<kTcN, TRB>(S.b, base + 3 * kTcABytes + TcFetch<kTcN, TRB>::place());
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic-proxy stores -> visible to the tensor core
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(T.full + 8 * st) : "memory");
}

// One thread of the last warp: the instructions of `total` slices, each when its stage is full, those of a run's first one
// when the run before has been drained.  RUN: slices of a run; 0: one run takes all.
template <bool TRA, bool TRB, int RUN>
__device__ __forceinline__ void tc_issue(TcCta& T, const int total)
{
    constexpr uint32_t idesc = tc_idesc<TRA, TRB>();
    constexpr uint64_t pa = kTcABytes >> 4, pb = kTcBBytes >> 4;      // from part to part, in descriptor units of 16 bytes
    const uint32_t small = T.tmem + kTcAcc * kTcN;
    constexpr uint32_t accs = RUN > 0 ? kTcAcc - 1 : kTcAcc;
    uint32_t in_run = 0, runs = 0;
    for (uint32_t s = 0; s < (uint32_t)total; s++) {
        const uint32_t round = s / kTcStages, st = s - round * kTcStages;
        if (RUN > 0 && in_run == RUN) {
            in_run = 0;
            if (!tc_wait(T.drained, runs++ & 1)) T.failed = true;
        }
        if (!tc_wait(T.full + 8 * st, round & 1)) T.failed = true;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t base = smem_u32(T.stage) + st * kTcStageBytes;
        const uint64_t a0 = tc_smem_desc<TRA>(base), b0 = tc_smem_desc<TRB>(base + 3 * kTcABytes);
#pragma unroll
        for (uint32_t k = 0; k < kTcKc / 16; k++) {
            const uint64_t a = a0 + k * tc_kstep(TRA), b = b0 + k * tc_kstep(TRB);
            const uint32_t n = in_run * (kTcKc / 16) + k;
            tc_mma(T.tmem + (n % accs) * kTcN, a, b, idesc, n >= accs ? 1u : 0u);
            tc_mma(small, a, b + pb, idesc, n > 0 ? 1u : 0u);
            tc_mma(small, a + pa, b, idesc, 1u);
            tc_mma(small, a + pa, b + pb, idesc, 1u);
            tc_mma(small, a, b + 2 * pb, idesc, 1u);
            tc_mma(small, a + 2 * pa, b, idesc, 1u);
        }
        in_run++;
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(T.empty + 8 * st) : "memory");
    }
}

// 16 accumulator columns of this thread's row, from column `col` of tensor memory
__device__ __forceinline__ void tc_load16(uint32_t (&r)[16], uint32_t tmem, int col)
{
    const uint32_t addr = tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + (uint32_t)col;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr) : "memory");
}

__device__ __forceinline__ void tc_load8(uint32_t (&r)[8], uint32_t addr)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
}

// waits for the loads; the loaded values must not be used, or moved, before that
__device__ __forceinline__ void tc_loaded(uint32_t (&a)[8], uint32_t (&b)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) asm volatile("" : "+r"(a[i]), "+r"(b[i]));
}

// The eight warps that bring operands, once they have stored the second slice of the run behind it (the tensor core has done
// with this one by then, and has two more slices to go on with): adds run `run` to the sum so far, which lies in the third
// accumulator's place.  Rows and columns of a warp as in tc_finish.
template <int RUN>
__device__ __forceinline__ void tc_drain(TcCta& T)
{
    const uint32_t run = T.runs_drained++, s = (run + 1) * RUN - 1;
    if (!tc_wait(T.empty + 8 * (s % kTcStages), (s / kTcStages) & 1)) T.failed = true;
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t base = T.tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + (threadIdx.x >> 7) * 32;
#pragma unroll 1
    for (uint32_t addr = base; addr < base + 32; addr += 8) {
        uint32_t u[8], v[8], w[8];                              // (two at a time: the slices in flight take the registers)
        tc_load8(u, addr);
        tc_load8(v, addr + kTcN);
        tc_loaded(u, v);
#pragma unroll
        for (int i = 0; i < 8; i++) u[i] = __float_as_uint(__uint_as_float(u[i]) + __uint_as_float(v[i]));
        tc_load8(v, addr + kTcAcc * kTcN);
        tc_load8(w, addr + 2 * kTcN);                           // the sum so far; in the first run of no meaning
        tc_loaded(v, w);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float x = __uint_as_float(u[i]) + __uint_as_float(v[i]);
            u[i] = __float_as_uint(run > 0 ? __uint_as_float(w[i]) + x : x);
        }
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(addr + 2 * kTcN),
                     "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]) : "memory");
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(T.drained) : "memory");
}

// the run that is to be drained behind the slice just stored, if there is one
template <int RUN>
__device__ __forceinline__ void tc_drain_due(TcCta& T)
{
    if constexpr (RUN > 0)
        if (T.slices_done == (T.runs_drained + 1) * RUN + 2) tc_drain<RUN>(T);
}

// Waits for the last slice (its commit covers every instruction issued before it), adds the accumulators and leaves the tile
// in shared memory: row r at tile + r * kTcTileLd.  Returns it after a block barrier, tensor memory freed.  exact(m, n):
// the element in plain FP32, for tiles with results that are not finite.
template <int RUN, class Exact>
__device__ __forceinline__ float4* tc_finish(TcCta& T, const int total, Exact&& exact)
{
    float4* tile = reinterpret_cast<float4*>(T.stage);
    const int row = ((threadIdx.x >> 5) & 3) * 32 + (threadIdx.x & 31), half = threadIdx.x >> 7;
    const bool brings = threadIdx.x < kTcThreads;
    if constexpr (RUN > 0)                                      // a last run of one slice has not drained the one before it
        if (brings && (int)(T.runs_drained + 1) * RUN < total) tc_drain<RUN>(T);
    if (total > 0) {
        const uint32_t s = total - 1;
        if (!tc_wait(T.empty + 8 * (s % kTcStages), (s / kTcStages) & 1)) T.failed = true;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();                                            // every warp knows that the stages are free
    float seen = 0.f;                                           // of this thread's outputs: finite when they are (or wrongly not)
    if (brings && total > 0) {
#pragma unroll 1
        for (int c = 0; c < 2; c++) {
            const int c0 = half * 32 + c * 16;
            uint32_t u[kTcAcc + 1][16];
#pragma unroll
            for (int a = 0; a <= kTcAcc; a++) tc_load16(u[a], T.tmem, a * kTcN + c0);
            // the loaded values must not be used, or moved, before this wait
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int a = 0; a <= kTcAcc; a++)
#pragma unroll
                for (int i = 0; i < 16; i++) asm volatile("" : "+r"(u[a][i]));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int x = 4 * q + i;
                    // (a contraction of one slice of 32 has used two of the three accumulators; behind several runs this is
                    // the sum of all but the last)
                    const float third = total > (RUN > 0 ? RUN : 1) ? __uint_as_float(u[2][x]) : 0.f;
                    v[i] = ((__uint_as_float(u[0][x]) + __uint_as_float(u[1][x])) + third) + __uint_as_float(u[3][x]);
                    seen += v[i];
                }
                tile[row * kTcTileLd + (c0 >> 2) + q] = make_float4(v[0], v[1], v[2], v[3]);
            }
        }
    }
    const bool bad = __syncthreads_or(!(fabsf(seen) <= 3.4e38f));
    if (brings && (total == 0 || bad)) {
        for (int q = 0; q < 8; q++) {
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (bad)
                for (int i = 0; i < 4; i++) v[i] = exact(row, half * 32 + 4 * q + i);
            tile[row * kTcTileLd + half * 8 + q] = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
    if (T.failed) atomicOr(&g_status, CFB200_ST_TC_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((threadIdx.x >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(T.tmem), "r"((uint32_t)kTcCols) : "memory");
    return tile;
}

// ---- C = sum_s A_s op(B_s) (+ bias) (+ residual), ReLU / mask: same contract as gemm_kernel (linear.cu) ----------
template <bool B_KN, int RUN>
__global__ void __launch_bounds__(kTcBlock, 2) tc_gemm_kernel(const GemmBatch Gb)
{
    extern __shared__ uint8_t tc_smem[];
    __shared__ uint64_t mbar_slots[kTcBarriers];
    __shared__ uint32_t tmem_slot;
    const GemmArgs& G = Gb.g[blockIdx.z / Gb.splits];
    const int rank = blockIdx.z % Gb.splits;
    const int m0 = blockIdx.x * kTcM, n0 = blockIdx.y * kTcN;
    int total = 0;
    for (int s = 0; s < G.nseg; s++) total += G.seg[s].K / kTcKc;
    const int first = total * rank / Gb.splits;                 // this block's share of the slices
    total = total * (rank + 1) / Gb.splits - first;
    // the slices one after the other, over the segments; two register sets keep a slice's loads in flight behind the one in
    // work
    TcFetch<kTcM, false> FA;
    TcFetch<kTcN, B_KN> FB;
    int seg = 0, in_seg = first, ahead = 0;                     // the slice to fetch next: segment, number in it, number
    while (in_seg >= G.seg[seg].K / kTcKc) in_seg -= G.seg[seg++].K / kTcKc;
    auto open = [&]() {
        const GemmSeg& S = G.seg[seg];
        FA.open(S.A, S.lda, m0, G.M, in_seg * kTcKc, S.K);
        FB.open(S.B, S.ldb, n0, G.N, in_seg * kTcKc, S.K);
    };
    open();
    auto fetch = [&](TcSlice& R) {
        if (ahead++ >= total) return;
        if (in_seg == G.seg[seg].K / kTcKc) { seg++; in_seg = 0; open(); }
        FA.next(R.a);
        FB.next(R.b);
        in_seg++;
    };
    TcSlice R0, R1;
    const bool brings = threadIdx.x < kTcThreads;
    TcCta T;
    tc_begin(T, tc_smem, mbar_slots, &tmem_slot);
    wait_for_predecessors();
    if (brings) { fetch(R0); fetch(R1); }
    if (brings) {
        for (int s = 0; s < total; s += 2) {
            tc_slice<false, B_KN>(T, R0); fetch(R0); tc_drain_due<RUN>(T);
            if (s + 1 < total) { tc_slice<false, B_KN>(T, R1); fetch(R1); tc_drain_due<RUN>(T); }
        }
    } else if (threadIdx.x == kTcThreads) {
        tc_issue<false, B_KN, RUN>(T, total);
    }
    __syncwarp();
    float4* tile = tc_finish<RUN>(T, total, [&](const int r, const int c) {
        float v = 0.f;
        const int m = m0 + r, n = n0 + c;
        if (m >= G.M || n >= G.N) return v;
        for (int x = first; x < first + total; x++) {
            int s = 0, k0 = x;
            while (k0 >= G.seg[s].K / kTcKc) { k0 -= G.seg[s].K / kTcKc; s++; }
            const GemmSeg& S = G.seg[s];
            for (int k = k0 * kTcKc; k < (k0 + 1) * kTcKc; k++)
                v = fmaf(__ldg(S.A + (size_t)m * S.lda + k), __ldg(B_KN ? S.B + (size_t)k * S.ldb + n : S.B + (size_t)n * S.ldb + k), v);
        }
        return v;
    });
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, n = n0 + 4 * tx;
    const bool stores = threadIdx.x < kTcThreads;
    if (Gb.splits == 1) {
        if (!stores) return;
#pragma unroll 4
        for (int r = ty; r < kTcM; r += kTcThreads / 16) gemm_finish(G, m0 + r, n, tile[r * kTcTileLd + tx]);
        return;
    }
    // the blocks' partial tiles lie in their shared memories; each block finishes its share of the rows
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
#pragma unroll 2
    for (int r = kTcM * rank / Gb.splits + ty; stores && r < kTcM * (rank + 1) / Gb.splits; r += kTcThreads / 16) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < Gb.splits; k++) {
            const float4 u = cluster.map_shared_rank(tile, k)[r * kTcTileLd + tx];
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        gemm_finish(G, m0 + r, n, v);
    }
    cluster.sync();                                             // no block leaves while its tile is being read
}

// Whether the tensor cores take a batch: whole slices and tiles, enough rows, and a result that does not depend on how its
// sums are formed.  Up to some 400 rows both kernels are one chain of latencies, and this one's is the longer (7.5 against
// 7.1 us); at 600 rows and [128] -> [512] it takes 7.6 against 10.3.
constexpr int kTcMinRows = 512;
static bool tc_gemm_covers(const GemmBatch& Gb)
{
    if (Gb.whole || Gb.g[0].M < kTcMinRows) return false;
    for (int i = 0; i < Gb.n; i++) {
        if (Gb.g[i].N % kTcN) return false;
        for (int s = 0; s < Gb.g[i].nseg; s++)
            if (Gb.g[i].seg[s].K % kTcKc) return false;
    }
    return true;
}

static int tc_slices(const GemmArgs& G)
{
    int slices = 0;
    for (int s = 0; s < G.nseg; s++) slices += G.seg[s].K / kTcKc;
    return slices;
}

template <bool B_KN, int RUN>
static int launch_tc_gemm(GemmBatch& Gb, cudaStream_t st)
{
    const GemmArgs& G = Gb.g[0];
    auto kern = tc_gemm_kernel<B_KN, RUN>;
    static std::atomic<bool> attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemBytes) != cudaSuccess) return CFB200_E_CUDA;
        attr_done[dev & 63] = true;
    }
    const int slices = tc_slices(G);
    const unsigned gx = (unsigned)((G.M + kTcM - 1) / kTcM), gy = (unsigned)(G.N / kTcN);
    // blocks that share a tile's contraction: as many as have four slices each, up to four, while all are resident at once
    int splits = slices / 4 < 4 ? slices / 4 : 4;
    while (splits > 1 && (int64_t)gx * gy * Gb.n * splits > 2 * (int64_t)sm_count()) splits--;
    Gb.splits = splits < 1 ? 1 : splits;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gx, gy, (unsigned)(Gb.n * Gb.splits));
    cfg.blockDim = dim3(kTcBlock);
    cfg.dynamicSmemBytes = kTcSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // as launch_ahead
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = (unsigned)Gb.splits;
    cfg.attrs = attr;
    cfg.numAttrs = Gb.splits > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, (const GemmBatch)Gb) == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

static int tc_gemm_batch(GemmBatch& Gb, bool b_kn, cudaStream_t st)
{
    bool whole = true;
    for (int i = 0; i < Gb.n; i++) whole = whole && tc_slices(Gb.g[i]) <= kTcWholeGemm;
    if (whole) return b_kn ? launch_tc_gemm<true, 0>(Gb, st) : launch_tc_gemm<false, 0>(Gb, st);
    return b_kn ? launch_tc_gemm<true, kTcRunGemm>(Gb, st) : launch_tc_gemm<false, kTcRunGemm>(Gb, st);
}

// ---- weight gradients: out[P,Q] = A[M,P]^T B[M,Q], rows split over gridDim.y, partial tiles to scratch -------
// Same problem table, scratch layout and reduction as wgrad_kernel (linear.cu); tiles are 128 x 64 and both operands are
// staged transposed (the contraction index, the atom, is the slow index of A and B in memory).
template <int RUN>
__global__ void __launch_bounds__(kTcBlock, 2) tc_wgrad_kernel(const WgArgs W)
{
    extern __shared__ uint8_t tc_smem[];
    __shared__ uint64_t mbar_slots[kTcBarriers];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x;
    int pi = 0;
    while (pi + 1 < W.nprob && (int)blockIdx.x >= W.prob[pi + 1].tile0) pi++;
    const WgProblem& Pb = W.prob[pi];
    const int t = blockIdx.x - Pb.tile0;
    const int p0 = (t / Pb.tiles_q) * kTcM, q0 = (t % Pb.tiles_q) * kTcN;
    const int split = blockIdx.y;
    const int r0 = split * W.rows, r1 = min(W.M, r0 + W.rows);
    const bool want_bias = Pb.bias_out != nullptr && q0 == 0;
    const int total = r1 > r0 ? (r1 - r0 + kTcKc - 1) / kTcKc : 0;
    TcFetch<kTcM, true> FA;
    TcFetch<kTcN, true> FB;
    FA.open(Pb.A, Pb.lda, p0, Pb.P, r0, r1);
    FB.open(Pb.B, Pb.ldb, q0, Pb.Q, r0, r1);
    auto fetch = [&](TcSlice& R) { FA.next(R.a); FB.next(R.b); };       // rows beyond r1 read as zeros
    float4 col = make_float4(0.f, 0.f, 0.f, 0.f);               // column sums of A over this thread's rows of the batch (the
    static_assert(kTcThreads % (kTcM / 4) == 0, "");             // float4 of a thread lie in the same columns)
    TcCta T;
    auto step = [&](const TcSlice& R) {
        if (want_bias) {
#pragma unroll
            for (int i = 0; i < tc_float4(kTcM); i++) { col.x += R.a[i].x; col.y += R.a[i].y; col.z += R.a[i].z; col.w += R.a[i].w; }
        }
        tc_slice<true, true>(T, R);
    };
    TcSlice R0, R1;
    const bool brings = tid < kTcThreads;
    if (brings) { fetch(R0); fetch(R1); }
    tc_begin(T, tc_smem, mbar_slots, &tmem_slot);
    if (brings) {
        for (int s = 0; s < total; s += 2) {
            step(R0); fetch(R0); tc_drain_due<RUN>(T);
            if (s + 1 < total) { step(R1); fetch(R1); tc_drain_due<RUN>(T); }
        }
    } else if (tid == kTcThreads) {
        tc_issue<true, true, RUN>(T, total);
    }
    __syncwarp();
    const float4* tile = tc_finish<RUN>(T, total, [&](const int p, const int q) {
        float v = 0.f;
        for (int r = r0; r < r1; r++) v = fmaf(__ldg(Pb.A + (size_t)r * Pb.lda + p0 + p), __ldg(Pb.B + (size_t)r * Pb.ldb + q0 + q), v);
        return v;
    });
    float* ws = W.ws + Pb.ws_off + (size_t)split * Pb.P * Pb.Q;
#pragma unroll 4
    for (int r = tid >> 4; brings && r < kTcM; r += kTcThreads / 16)
        *reinterpret_cast<float4*>(ws + (size_t)(p0 + r) * Pb.Q + q0 + 4 * (tid & 15)) = tile[r * kTcTileLd + (tid & 15)];
    if (want_bias) {
        // threads tid, tid + 32, ... hold the same columns: eight partial sums beside the tile
        float4* part = const_cast<float4*>(tile) + kTcM * kTcTileLd;
        if (brings) part[tid] = col;
        __syncthreads();
        if (tid < kTcM / 4) {
            float4 v = part[tid];
#pragma unroll
            for (int w = 1; w < kTcThreads * 4 / kTcM; w++) { const float4 u = part[tid + w * (kTcM / 4)]; v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w; }
            float* o = W.ws + Pb.ws_off + (size_t)W.S * Pb.P * Pb.Q + (size_t)split * Pb.P + p0 + 4 * tid;
            o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
        }
    }
}

// whether the tensor cores take a weight gradient: whole tiles, enough rows
static bool tc_wgrad_covers(const WgProblem& Pb, int64_t M)
{
    return M >= kTcMinRows && Pb.nb == 1 && Pb.P % kTcM == 0 && Pb.Q % kTcN == 0;
}

template <int RUN>
static int launch_tc_wgrad(const WgArgs& W, int tiles, cudaStream_t st)
{
    static std::atomic<bool> attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63]) {
        if (cudaFuncSetAttribute(tc_wgrad_kernel<RUN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemBytes) != cudaSuccess) return CFB200_E_CUDA;
        attr_done[dev & 63] = true;
    }
    tc_wgrad_kernel<RUN><<<dim3(tiles, W.S), kTcBlock, kTcSmemBytes, st>>>(W);
    return cudaGetLastError() == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

static int tc_wgrad_launch(const WgArgs& W, int tiles, cudaStream_t st)
{
    return W.rows <= kTcWholeWgrad * kTcKc ? launch_tc_wgrad<0>(W, tiles, st) : launch_tc_wgrad<kTcRunWgrad>(W, tiles, st);
}

}  // namespace cfb
