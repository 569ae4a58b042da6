// Periodic attention of one encoder layer as two kernels: lattice-sum bias, frame-projected value
// encoding and ragged softmax attention together, forward and backward (what
// RealEncodingWithFramedProjFuncCUDA followed by FusedDotProductAttentionCUDA compute in the reference,
// models/indexed_lattice_multi_head_attention_cuda.py:944-985).
//
// The value encoding is linear in the 256 basis sums of a pair, values_ij = W s_ij, so the attention
// output  out_i = sum_j p_ij (v_j + W s_ij) = sum_j p_ij v_j + W (sum_j p_ij s_ij)  needs the 16 x 256
// projection once per (atom, head) instead of once per (pair, head), and the (E,H,16) value encoding and
// its gradient never exist in memory.  Backward likewise: W^T gout_i is formed once per (atom, head), the
// weight gradient is  sum_i gout_i (x) S_i  with the pooled basis S_i = sum_j p_ij s_ij saved by the
// forward (a small GEMM left to the caller), and the coefficient gradient of an atom is accumulated by
// the warp that walks its pairs -- no scratch, no second-stage reductions.
//
// Work decomposition: grid = (resident blocks, heads); warp = one (atom, head) at a time, taking the
// atom's pairs in tiles of 32 with an online softmax.  The cost of an atom varies a hundredfold (1 to 64+ pairs, a few
// to a hundred surviving translations each), so warps draw atoms from a per-head queue in the order given
// by ``order`` (most expensive first).  Which warp computes an atom does not affect any result: nothing is
// accumulated across atoms, so every sum stays deterministic.  Outputs of the forward: out (N,H,16), z (E,H), lse (N,H), spool (N,H,256) with the
// distance part unscaled and the angle parts times the angle coefficient (the scaling the reference's
// weight gradients carry).  The backward leaves gz (E,H) for the column pass that forms gk and gv
// (dpa_bwd_cols_kernel), gq (N,H,16) with respect to the scaled query, and ga (N,H).
//
// Chunked queue (kernels instantiated with TASKS): one warp walks the pairs of an (atom, head) one after the other, so an
// atom of a dense 64-atom cell with a wide Gaussian can take several times a warp's average load and the launch
// would end with that warp alone.  attn_plan_kernel turns the batch's work queue (atom_order_kernel) and the layer's
// coefficients into a table of tasks per head: an atom whole, or one chunk of its pairs.  A chunk is computed exactly
// like an atom with fewer pairs and leaves its result in a partial row; attn_merge_fwd / _bwd_kernel combine the
// rows of an atom in chunk order (softmax-weighted by the chunks' log-sum-exp; plain sums backward), so results do
// not depend on which warp ran what.
#include <atomic>
#include "lattice_lane.cuh"

namespace cfb {

constexpr int kAtHd = 16;
constexpr int kAtK = 256;

struct AtArgs {
    const float* qs; const float* k; const float* v; const float* a_ik;
    const float* pos_ij; const float* tvecs; const float* rvlen;
    const int64_t* batch; const int64_t* edges; const int64_t* e_start; const int32_t* order;
    int* counters;            // (H) work-queue heads, zeroed before the launch
    int counters_zeroed;      // they already are
    int pairwise;             // forward that leaves per-pair results: one pair after the other (attn_pairwise_kernel)
    // task table of the chunked queue (attn_plan_kernel), or NULL: then ``order`` (or the atom index) is the queue
    const int4* tasks; int64_t n_entries;
    int* chunk_count;         // (H) chunk entries in use per head: they sit at the end of the chunk region
    float* part_out; float* part_lse; float* part_spool;               // forward results of chunks (kSplitSlots rows)
    float* part_gq; float* part_ga;                                    // backward results of chunks
    int64_t N, E;
    const float* W[4]; const float* frame[3];
    const float* list; int cache_range;
    int vec, vec_list;        // q, k, val, gout and v are 16-byte aligned: 128-bit loads, 64-bit stores; the lists are
    float* z; float* out; float* lse; float* spool;                    // forward outputs
    const float* gout; const float* z_in;                             // backward inputs (plus out, lse above)
    float* gz; float* gq; float* ga;                                   // backward outputs
    // what a training forward leaves for a backward pass without a second lattice sum: per pair its value encoding
    // (E,H,16) and sum p d^2 (E,H); per atom the projection of the attention-pooled d^2-weighted basis sums (N,H,16)
    float* val; float* px; float* upool;
    float* part_upool;                                                  // its chunk results (kSplitSlots rows)
};

// next atom of this head's work queue (one atomic per task; the whole warp gets the same answer)
__device__ __forceinline__ int64_t next_task(int* counter, const int lane)
{
    int t = 0;
    if (lane == 0) t = atomicAdd(counter, 1);
    return (int64_t)__shfl_sync(0xffffffffu, t, 0);
}

// ---- the kernel ------------------------------------------------------------------------------------------------
// What bounds it: instruction issue.  A pair keeps few translations (means over the batches of synth.py: 12 for cells
// of 3-10 A, 6 for the log-normal ones, 2 for cells of 10-25 A), so the fixed cost of a pair -- reading its list, three
// warp reductions, logarithm and exponentials, its 16 x 256 projection -- used to outweigh its translations (about
// 800 of 1 100 instructions).  Therefore
//   * lane = pair for everything that is per pair: normaliser, q.k, bias, soft-max weight (tiles of 32 pairs);
//   * the surviving translations of a tile are numbered through, and lane = translation makes their records 32 at a
//     time whatever pair they belong to;
//   * only the walk over the records runs with lane = basis index (l and l + 32 of each 64-wide basis), and only it
//     costs instructions per translation;
//   * where a pair's sums are kept they are projected four pairs at a time, so that a weight is read once for four;
//     else the pair's soft-max weight enters the pooled sums directly and there is no per-pair work in the walk at all.
// Both directions are this kernel: a backward pass that recomputes the lattice sums differs in what a translation's
// Gaussians are multiplied with (W^T gout of the atom, giving gout . W s_ij and gout . W t_ij per pair).
// Instructions per (pair, head): 256 log-normal crystals, forward 690, with per-pair results 1 050; eight cells of 100-200
// atoms, forward 127, backward 146.
// With s_ij the basis sums of a pair, t_ij the same sums weighted with d^2 and x_ij = sum p d^2, the backward pass is
//   gz_ij = p_ij (gout_i . (v_j + W s_ij) - gout_i . out_i)
//   ga_i  = sum_j c_dist x_ij gz_ij + p_ij gout_i . W (t_ij - x_ij s_ij)
//         = gout_i . W (sum_j p_ij t_ij) + sum_j (c_dist x_ij gz_ij - p_ij x_ij gout_i . W s_ij)
// so it needs the lattice sums only through the pair's value encoding W s_ij (16 numbers), x_ij, and the projection
// of the attention-pooled t of the atom (16 numbers per atom).  None of these depends on gout: the training forward
// leaves them (68 bytes per (pair, head)) and attn_bwd_saved_kernel is a plain ragged attention backward.

// AH: halves of 32 angle Gaussians per axis: 0 (no frames), 1 (angle_dim <= 32), 2
__host__ __device__ constexpr int fw_k(int AH) { return 64 + 96 * AH; }        // basis indices a row holds
constexpr int kFwRec = 12;                  // floats per record (8 used): conflict-free 128-bit writes
constexpr int kFwWait = 8, kFwWaitLd = 33;  // backward: pairs whose lane sums wait for the reduction over the lanes; stride
constexpr int kFwStage = 64;                // translations of an unlisted pair that wait for their records
// MODE 0: forward.  1: forward that leaves per-pair results.  2: backward without them.
__host__ __device__ constexpr int fw_rows(int mode) { return mode == 1 ? 4 : (mode == 0 ? 1 : 0); }
// warps per block and resident blocks per SM: 64, 96 and 80 registers per thread.  Mode 2, 256 log-normal crystals: 6 x 4
// 228 us, 12 x 2 242 us; mode 1: 10 x 2 335 us, 5 x 4 352 us, 12 x 2 (80 registers) 374 us; mode 0: within 2 %.
__host__ __device__ constexpr int fw_warps(int mode) { return mode == 0 ? 16 : (mode == 1 ? 10 : 6); }
__host__ __device__ constexpr int fw_blocks(int mode) { return mode == 2 ? 4 : 2; }
// EACH: mode 2 with lane sums formed pair by pair (see drain)
__host__ __device__ constexpr size_t fw_smem_bytes(int AH, int mode, bool each)
{
    return sizeof(float) * (kAtHd * fw_k(AH) + fw_warps(mode) * (32 * kFwRec + 5 * kFwStage + fw_rows(mode) * fw_k(AH) +
                                                                      (mode == 2 && !each ? 2 * kFwWait * kFwWaitLd : 0)));
}
// translations whose weight is below exp(-24) = 4e-11 of the nearest one's do not enter the normaliser: the 125 of a
// box together stay below a tenth of its last bit
constexpr float kFwCut = 24.0f;
// The backward without lists weighs translations against their sum and not against the nearest one: log(125) apart at most
// in a box of two cells each way.
constexpr float kFwLogBox = 4.83f;
// Where no per-pair results are wanted, the translations of a pair with a faint soft-max weight are not walked.  Forward:
// below exp(-24) of its atom's largest so far; it adds nothing to the atom's sums that their last bit could hold (200 such
// pairs together 1e-8 of one with the largest weight).  Backward: below exp(-24) of the sum over the atom's pairs; its gz_ij
// loses the part p gout . W s_ij, an absolute error of at most exp(-24) |gout . W s_ij|, which gk_j and gq_i take on times
// a query's and a key's size, and ga_i times x_ij.  The bias of such a pair enters the soft-max like every other's.  In cells of 10-25 A a
// quarter of the pairs are that far apart: 64 crystals of 100-200 atoms, forward 1.80 -> 1.37 ms
// (1.53 with the pooled sums in shared memory), backward 2.81 -> 2.04.
constexpr float kFwFaint = 3.7751345e-11f;       // exp(-24)

// W . row for R rows: lane = (outputs 4 g .. 4 g + 3 with g = l >> 3, eighth l & 7 of every 32 basis indices).  Returns
// two outputs of one row: of row fw_row(l), from output fw_out(l) on.  Packed FP32: two products per instruction, two
// partial sums.  A 128-bit shared-memory read costs its bytes per lane however many lanes share an address, so the
// block of outputs per lane is made as square as the registers allow: 16 outputs from 8 reads per 4 basis indices.
__device__ __forceinline__ int fw_row(const int lane) { return (lane >> 1) & 3; }
__device__ __forceinline__ int fw_out(const int lane) { return 4 * (lane >> 3) + 2 * (lane & 1); }

template <int AH, int R>
__device__ __forceinline__ float2 fw_project(const float* W_s, const float* rows, const int lane)
{
    constexpr int K = fw_k(AH);
    const int g = lane >> 3, kc = lane & 7;
    const ulonglong2* w0 = reinterpret_cast<const ulonglong2*>(W_s + 4 * g * K) + kc;
    const ulonglong2* r0 = reinterpret_cast<const ulonglong2*>(rows) + kc;
    f32x2 acc[R][4];
#pragma unroll
    for (int r = 0; r < R; r++) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = pack2(0.f, 0.f);
#pragma unroll 1
    for (int s = 0; s < K / 32; s++) {
        ulonglong2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = r0[r * (K / 4) + 8 * s];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const ulonglong2 w = w0[c * (K / 4) + 8 * s];
#pragma unroll
            for (int r = 0; r < R; r++) {
                acc[r][c] = fma2(v[r].x, w.x, acc[r][c]); acc[r][c] = fma2(v[r].y, w.y, acc[r][c]);
            }
        }
    }
    float o[R][4];
#pragma unroll
    for (int r = 0; r < R; r++) {
#pragma unroll
        for (int c = 0; c < 4; c++) { float x, y; unpack2(acc[r][c], x, y); o[r][c] = x + y; }
    }
    // the eighths are summed; a lane passes on the rows and outputs it does not keep
    float q[4];
    if constexpr (R == 4) {
        const bool up4 = kc & 4, up2 = kc & 2;
        float h[2][4];
#pragma unroll
        for (int r = 0; r < 2; r++) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float send = up4 ? o[r][c] : o[r + 2][c], keep = up4 ? o[r + 2][c] : o[r][c];
                h[r][c] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float send = up2 ? h[0][c] : h[1][c], keep = up2 ? h[1][c] : h[0][c];
            q[c] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                o[r][c] += __shfl_xor_sync(0xffffffffu, o[r][c], 4);
                o[r][c] += __shfl_xor_sync(0xffffffffu, o[r][c], 2);
            }
            q[c] = R > 1 && fw_row(lane) == 1 ? o[R - 1][c] : o[0][c];
        }
    }
    const bool up1 = kc & 1;
    const float s0 = up1 ? q[0] : q[2], s1 = up1 ? q[1] : q[3];
    float2 out;
    out.x = (up1 ? q[2] : q[0]) + __shfl_xor_sync(0xffffffffu, s0, 1);
    out.y = (up1 ? q[3] : q[1]) + __shfl_xor_sync(0xffffffffu, s1, 1);
    return out;
}

// What a lane of the walk knows of the bases.  Windows, one byte per basis (distance, three axes): with lo the first index
// inside, this lane's index l is inside when l >= lo and l <= lo + win - 1, and l + 32 when l + 32 >= lo and l + 32 <=
// lo + win - 1.  Each comparison is bit 6 of a byte of a packed difference biased by 64 (no byte leaves 0..127), so that four
// additions and two ANDs serve the four bases.
struct FwLane {
    unsigned in0_lo, in0_hi, in1_lo, in1_hi;
    float cd_lo, cd_hi, nca_lo, nca_hi;      // basis constants, pre-scaled so that a Gaussian is ex2(-b*b)
    float d0, dstep, a0, nastep;             // the same as number of the lane's first index, and step
    bool wide_d;
    __device__ __forceinline__ FwLane(const Params& P, const int lane)
    {
        const unsigned lane4 = lane * 0x01010101u;
        const unsigned wins = (unsigned)P.win_dist | (unsigned)P.win_ang * 0x01010100u;
        in0_lo = 0x40404040u + lane4; in0_hi = 0x3F3F3F3Fu + wins - lane4;
        in1_lo = 0x60606060u + lane4; in1_hi = 0x1F1F1F1Fu + wins - lane4;
        const float astep = P.a_step * kLlSqrtLog2e;
        dstep = P.d_step * kLlSqrtLog2e; nastep = -astep;
        d0 = (float)(lane + 1); a0 = (float)(P.angle_dim - 1 - lane);
        cd_lo = (float)(lane + 1) * dstep; cd_hi = (float)(lane + 33) * dstep;
        nca_lo = -(float)(P.angle_dim - 1 - lane) * astep; nca_hi = -(float)(P.angle_dim - 33 - lane) * astep;
        wide_d = P.win_dist > 32;
    }
};

// the record of a translation with weight exp(arg) relative to the pair's nearest, for (atom, head) ih; third: what the
// walk multiplies its Gaussians with
template <int AH>
__device__ __forceinline__ void fw_record(const AtArgs& A, const Params& P, const int64_t ih, float* dst, const float arg, const float d2,
                                          const float dx, const float dy, const float dz, const float third, const int flag)
{
    // d and 1/d from one reciprocal square root plus a Newton step; quotients by the basis spacings
    // become products with their reciprocals (last-bit differences from IEEE sqrt / division)
    float rinv = rsqrtf(fmaxf(d2, 1e-30f));
    rinv = rinv * fmaf(-0.5f * d2 * rinv, rinv, 1.5f);
    const float d = d2 * rinv;
    int lo_d = 0;
    if (P.windowed_dist) {
        lo_d = (int)(fmaf(d, P.inv_d_interval, -P.d_cut_scaled) - 1.0f);
        lo_d = min(max(lo_d, 0), 64 - P.win_dist);
    }
    float xa[3] = {0.f, 0.f, 0.f};
    int lo_pack = lo_d;
    if constexpr (AH > 0) {
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const float* F = A.frame[x] + ih * 3;
            float cosv = 1e3f;
            if (d2 > 1e-5f) cosv = fmaf(dz, __ldg(F + 2), fmaf(dy, __ldg(F + 1), dx * __ldg(F))) * rinv;
            if (P.cos_abs) cosv = fabsf(cosv);
            int lo = 0;
            if (P.windowed_ang) {
                const float en = fmaf(cosv + 1.0f + P.a_cut, P.inv_a_interval, 1.0f);
                int end = (int)fminf(en, (float)P.angle_dim);
                end = max(end, P.win_ang);
                lo = end - P.win_ang;
            }
            xa[x] = (1.0f - cosv) * P.xa_scale;
            lo_pack |= lo << (8 * (x + 1));
        }
    }
    // minus the log2 of the weight
    float4* o = reinterpret_cast<float4*>(dst);
    o[0] = make_float4(-(arg * kLlLog2e), -d * P.xd_scale, third, __int_as_float(flag));
    if constexpr (AH > 0) o[1] = make_float4(xa[0], xa[1], xa[2], __int_as_float(lo_pack));
    else o[1].x = __int_as_float(lo_pack);
}

// lane = basis index: the Gaussians, times the weight, of record R (u its first half) that fall on this lane: add(k, value),
// k as the lane numbers its indices (distance l, l + 32, axis 1 l, ...).  ONE_ROUNDING: a Gaussian's argument is the fused
// x + number * step, as the compiler forms it in LatticeLane, and not x + (rounded constant).
template <int AH, bool ONE_ROUNDING, class Add>
__device__ __forceinline__ void fw_gaussians(const FwLane& L, const float4* R, const float4& u, Add&& add)
{
    const float nlw = u.x, xd = u.y;
    float xa[3];
    unsigned lo;
    if constexpr (AH > 0) {
        const float4 v = R[1];
        xa[0] = v.x; xa[1] = v.y; xa[2] = v.z; lo = __float_as_uint(v.w);
    } else {
        lo = *reinterpret_cast<const unsigned*>(R + 1);
    }
    const unsigned in0 = (L.in0_lo - lo) & (L.in0_hi + lo), in1 = (L.in1_lo - lo) & (L.in1_hi + lo);
    if (!L.wide_d) {                                        // at most one of the lane's two indices is in the window
        const bool hi = in1 & 0x40u;
        const float b = ONE_ROUNDING ? fmaf(hi ? L.d0 + 32.0f : L.d0, L.dstep, xd) : xd + (hi ? L.cd_hi : L.cd_lo);
        const float g = ex2_approx(-fmaf(b, b, nlw));
        if (in0 & 0x40u) add(0, g);
        if (hi) add(1, g);
    } else {
        const float b0 = ONE_ROUNDING ? fmaf(L.d0, L.dstep, xd) : xd + L.cd_lo;
        const float b1 = ONE_ROUNDING ? fmaf(L.d0 + 32.0f, L.dstep, xd) : xd + L.cd_hi;
        const float g0 = ex2_approx(-fmaf(b0, b0, nlw)), g1 = ex2_approx(-fmaf(b1, b1, nlw));
        if (in0 & 0x40u) add(0, g0);
        if (in1 & 0x40u) add(1, g1);
    }
    if constexpr (AH > 0) {
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const float b0 = ONE_ROUNDING ? fmaf(L.a0, L.nastep, xa[x]) : xa[x] + L.nca_lo;
            const float g0 = ex2_approx(-fmaf(b0, b0, nlw));
            if (in0 & (0x4000u << (8 * x))) add(2 + AH * x, g0);
            if constexpr (AH == 2) {
                const float b1 = ONE_ROUNDING ? fmaf(L.a0 - 32.0f, L.nastep, xa[x]) : xa[x] + L.nca_hi;
                const float g1 = ex2_approx(-fmaf(b1, b1, nlw));
                if (in1 & (0x4000u << (8 * x))) add(3 + AH * x, g1);
            }
        }
    }
}

template <int AH, bool TASKS, int MODE, bool EACH>
__global__ void __launch_bounds__(fw_warps(MODE) * 32, fw_blocks(MODE)) attn_tile_kernel(const AtArgs A, const Params P)
{
    wait_for_predecessors();
    extern __shared__ __align__(16) float smem[];
    constexpr int K = fw_k(AH), RS = kFwRec, kWarps = fw_warps(MODE);
    constexpr bool SAVE = MODE == 1, BACK = MODE == 2;
    constexpr int NB = 1 + (AH == 0 ? 0 : 3);               // bases
    constexpr int NS = 2 + 3 * AH;                          // basis indices per lane
    float* W_s = smem;                                      // [16][K], scaled, lane-paired order (see rows)
    const int H = P.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* rec = W_s + kAtHd * K + warp * 32 * RS;         // this warp's records
    float* stage = W_s + kAtHd * K + kWarps * 32 * RS + warp * 5 * kFwStage;
    float* rows = W_s + kAtHd * K + kWarps * (32 * RS + 5 * kFwStage) + warp * fw_rows(MODE) * K;   // basis vectors to project: per basis
                                                            // (lane, half) pairs, or lanes where there is one half
    float2* wait = reinterpret_cast<float2*>(W_s + kAtHd * K + kWarps * (32 * RS + 5 * kFwStage)) + warp * kFwWait * kFwWaitLd;
    const FwLane L(P, lane);
    const float cut = fmaxf(P.prune, kFwCut);
    __shared__ int head_open;

    // A block serves its own head first and then, turn by turn, the head with the most entries left: the heads' Gaussian
    // widths differ, so their queues hold up to a fifth more or less work than the average, and the blocks of the light
    // heads would otherwise sit idle while the heaviest head finishes.  Switching heads costs a reload of the head's
    // projection weights.
    for (int turn = 0; turn < 2 * H; turn++) {
    int h = blockIdx.y;
    if (turn > 0) {
        __syncthreads();                                    // every warp is done with the previous head's weights
        if (threadIdx.x == 0) {
            // the head with the most entries left in its queue (a stale count costs a wasted or a missed turn at most)
            int best = -1, most = 0;
            for (int hh = 0; hh < H; hh++) {
                const int limit = TASKS ? (int)(A.n_entries - kSplitSlots) + __ldg(A.chunk_count + hh) : (int)A.N;
                const int left = limit - atomicAdd(A.counters + hh, 0);
                if (left > most) { most = left; best = hh; }
            }
            head_open = best;
        }
        __syncthreads();
        h = head_open;
        if (h < 0) break;                                   // every queue is drained
    }
    const int first = TASKS ? kSplitSlots - __ldg(A.chunk_count + h) : 0;
    for (int idx = threadIdx.x; idx < kAtHd * NB * 64; idx += kWarps * 32) {
        const int o = idx / (NB * 64), b = (idx >> 6) % NB, d = idx & 63;
        if (AH == 1 && b > 0 && d >= 32) continue;
        const int width = b == 0 ? 64 : P.angle_dim;        // columns this basis' weights hold (zero beyond)
        const float w = d < width ? __ldg(A.W[b] + ((size_t)h * kAtHd + o) * width + d) : 0.f;
        const int pos = b == 0 || AH == 2 ? 64 * b + 2 * (d & 31) + (d >> 5) : 64 + 32 * (b - 1) + d;
        W_s[o * K + pos] = w * (b == 0 ? P.c_dist : P.c_ang);
    }
    __syncthreads();

    for (;;) {
        const int64_t t = next_task(A.counters + h, lane) + first;
        if (t >= (TASKS ? A.n_entries : A.N)) break;
        int i, row;
        int off = 0, np;                                    // the task's pairs: np of them from the atom's pair off
        int64_t e0;
        if (TASKS) {
            const int4 d = __ldg(A.tasks + (size_t)h * A.n_entries + t);
            np = d.w & 0xFFFFFF;
            if (np == 0) continue;                          // an entry this head does not use
            i = d.x; row = d.y; off = d.z;
            e0 = A.e_start[i];
        } else {
            i = A.order != nullptr ? A.order[t] : (int)t;
            row = i;
            e0 = A.e_start[i];
            np = (int)(A.e_start[i + 1] - e0);
        }
        const int64_t ih = (int64_t)i * H + h;
        const int c = (int)A.batch[i];
        const float a = __ldg(A.a_ik + ih);
        int Rl = 0;
        if (lane < 3) Rl = lattice_range_1d(P, a, P.cutoff_radius != 0.0f ? __ldg(A.rvlen + 3 * (int64_t)c + lane) : 0.0f);
        const int R1 = __shfl_sync(0xffffffffu, Rl, 0), R2 = __shfl_sync(0xffffffffu, Rl, 1), R3 = __shfl_sync(0xffffffffu, Rl, 2);
        const bool use_list = A.list != nullptr && R1 == A.cache_range && R2 == A.cache_range && R3 == A.cache_range;
        // the pairs of an atom run over the atoms of its crystal in order: key atom = first atom + offset
        e0 += off;
        const int j0 = np > 0 ? (int)A.edges[A.E + e0] : 0;
        float m = -INFINITY, l = 0.f, V = 0.f;              // l: this lane's pairs; V: component l & 15, pairs of parity l >> 4
        // forward: sums of a pair, plain and (T) d^2-weighted, and both pooled with the attention weights (S, Tq): an addition
        // per pair, as one chain over all of an atom's terms would round three times as much.  Backward: S = W^T gout
        float s[NS], S[NS], T[SAVE ? NS : 1], Tq[SAVE ? NS : 1];
#pragma unroll
        for (int r = 0; r < NS; r++) { s[r] = S[r] = 0.f; if constexpr (SAVE) T[r] = Tq[r] = 0.f; }
        float D = 0.f, lse = 0.f, ga = 0.f;                 // backward: gout . out, log-sum-exp, coefficient gradient
        float cA = 0.f, cB = 0.f, accA = 0.f, accB = 0.f;   // backward: gout . W t and gout . W s, of lane's pair and in the making
        if constexpr (BACK) {
            float god = 0.f, od = 0.f;
            if (lane < kAtHd) {
                god = __ldg(A.gout + ih * kAtHd + lane);
                od = __ldg(A.out + ih * kAtHd + lane);
            }
            D = warp_sum(god * od);
            lse = __ldg(A.lse + ih);
#pragma unroll 4
            for (int o = 0; o < kAtHd; o++) {
                const float go = __shfl_sync(0xffffffffu, god, o);
                const float2 w = *reinterpret_cast<const float2*>(W_s + o * K + 2 * lane);
                S[0] = fmaf(go, w.x, S[0]); S[1] = fmaf(go, w.y, S[1]);
#pragma unroll
                for (int x = 0; x < NB - 1; x++) {
                    if constexpr (AH == 2) {
                        const float2 u = *reinterpret_cast<const float2*>(W_s + o * K + 64 + 64 * x + 2 * lane);
                        S[2 + 2 * x] = fmaf(go, u.x, S[2 + 2 * x]); S[3 + 2 * x] = fmaf(go, u.y, S[3 + 2 * x]);
                    } else if constexpr (AH == 1) {
                        S[2 + x] = fmaf(go, W_s[o * K + 64 + 32 * x + lane], S[2 + x]);
                    }
                }
            }
        }
        float inv = 0.f, f = 0.f;                           // lane = pair: 1 / normaliser, soft-max weight / normaliser
        int tile0 = 0;                                      // first pair of the tile

        // Forward without per-pair results: the pooled sums lie in this warp's row (a lane touches its own entries only) and
        // take up what up to 32 records gave.  One chain of additions over an atom's few hundred terms would cost a third
        // more rounding (out 2.2e-7 against 1.7e-7 of a 64-bit result for dense cells), and pooled sums in registers cost
        // 18 % of the time where these cost 11 % (16 crystals of 100-200 atoms: 407 us without, 484, 460).
        auto pooled = [&](auto&& f) {
            float2* p0 = reinterpret_cast<float2*>(rows + 2 * lane);
            const float2 u = *p0;
            *p0 = make_float2(f(0, u.x), f(1, u.y));
            if constexpr (AH == 2) {
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    float2* p = reinterpret_cast<float2*>(rows + 64 + 64 * x + 2 * lane);
                    const float2 w = *p;
                    *p = make_float2(f(2 + 2 * x, w.x), f(3 + 2 * x, w.y));
                }
            } else if constexpr (AH == 1) {
#pragma unroll
                for (int x = 0; x < 3; x++) rows[64 + 32 * x + lane] = f(2 + x, rows[64 + 32 * x + lane]);
            }
        };
        auto clear = [&]() {
#pragma unroll
            for (int k = 0; k < NS; k++) s[k] = 0.f;
        };
        if constexpr (MODE == 0) pooled([](const int, const float) { return 0.f; });

        // Backward: a pair's two sums over the lanes.  A butterfly per pair is seven dependent shuffles; eight pairs at once
        // (lane = pair, quarter of the lanes) are 30 instructions, and the sums go to the lanes that hold the pairs.  What either
        // gives depends on the instance (EACH: butterflies), us per launch, butterflies / eight at once.  Frames, task table: 64
        // cells of 100-200 atoms 1 992 / 1 936, 256 log-normal crystals 399 / 412; frames, no table, with the column pass: 2 103 /
        // 2 071, 511 / 513.  Plain, task table: 1 377 / 1 308, 16 cells 333 / 321, cells of 20-100 atoms 322 / 323, of 50 249 /
        // 244, but 256 log-normal crystals 220 / 238, 1 024 710 / 750, 256 of 4-16 atoms 209 / 225; plain, no table, with the
        // column pass: 1 505 / 1 499, 262 / 300, 769 / 843.
        int waiting_pairs = 0, slot = -1;
        auto drain = [&]() {
            __syncwarp();
            const float2* p = wait + (lane & 7) * kFwWaitLd + (lane >> 3) * 8;
            float2 x[8];
#pragma unroll
            for (int k = 0; k < 8; k++) x[k] = p[k];
            float b = ((x[0].x + x[1].x) + (x[2].x + x[3].x)) + ((x[4].x + x[5].x) + (x[6].x + x[7].x));
            float c2 = ((x[0].y + x[1].y) + (x[2].y + x[3].y)) + ((x[4].y + x[5].y) + (x[6].y + x[7].y));
            b += __shfl_xor_sync(0xffffffffu, b, 8); c2 += __shfl_xor_sync(0xffffffffu, c2, 8);
            b += __shfl_xor_sync(0xffffffffu, b, 16); c2 += __shfl_xor_sync(0xffffffffu, c2, 16);
            b = __shfl_sync(0xffffffffu, b, slot & 7); c2 = __shfl_sync(0xffffffffu, c2, slot & 7);
            if (slot >= 0) { cB = b; cA = c2; slot = -1; }
            waiting_pairs = 0;
            __syncwarp();
        };

        // the tile's pair j is complete: into the pooled sums, and into the row that waits for its projection
        auto flush = [&](const int j) {
            if constexpr (BACK) {
                if constexpr (EACH) {
                    // both sums over the lanes at once: the lower half of the warp takes B, the upper A
                    const bool up = lane & 16;
                    float r = (up ? accA : accB) + __shfl_xor_sync(0xffffffffu, up ? accB : accA, 16);
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
                    const float b = __shfl_sync(0xffffffffu, r, 0), c2 = __shfl_sync(0xffffffffu, r, 16);
                    if (lane == j) { cB = b; cA = c2; }
                    accA = accB = 0.f;
                    return;
                }
                // the lanes' parts wait in shared memory until eight pairs are complete
                wait[waiting_pairs * kFwWaitLd + lane] = make_float2(accB, accA);
                if (lane == j) slot = waiting_pairs;
                accA = accB = 0.f;
                if (++waiting_pairs == kFwWait) drain();
                return;
            }
            const float fj = __shfl_sync(0xffffffffu, f, j), ij = __shfl_sync(0xffffffffu, inv, j);
            float* w = rows + (j & 3) * K;
            *reinterpret_cast<float2*>(w + 2 * lane) = make_float2(s[0] * ij, s[1] * ij);
            if constexpr (AH == 2) {
#pragma unroll
                for (int x = 0; x < 3; x++)
                    *reinterpret_cast<float2*>(w + 64 + 64 * x + 2 * lane) = make_float2(s[2 + 2 * x] * ij, s[3 + 2 * x] * ij);
            } else if constexpr (AH == 1) {
#pragma unroll
                for (int x = 0; x < 3; x++) w[64 + 32 * x + lane] = s[2 + x] * ij;
            }
#pragma unroll
            for (int r = 0; r < NS; r++) {
                S[r] = fmaf(fj, s[r], S[r]); s[r] = 0.f;
                if constexpr (SAVE) { Tq[r] = fmaf(fj, T[r], Tq[r]); T[r] = 0.f; }
            }
            if ((j & 3) == 3 || tile0 + j == np - 1) {
                __syncwarp();
                const float2 o = fw_project<AH, 4>(W_s, rows, lane);
                if (fw_row(lane) <= (j & 3)) {
                    float* dst = A.val + ((e0 + tile0 + (j & ~3) + fw_row(lane)) * H + h) * kAtHd + fw_out(lane);
                    if (A.vec) *reinterpret_cast<float2*>(dst) = o;
                    else { dst[0] = o.x; dst[1] = o.y; }
                }
                __syncwarp();
            }
        };

        // lane = translation: the record of a translation with weight exp(arg) relative to the pair's nearest
        auto make_record = [&](const int slot, const float arg, const float d2, const float dx, const float dy, const float dz,
                               const float fj, const int flag) {
            // third: the soft-max weight forward (d^2 where a pair's sums are kept); d^2 less the nearest one's (fj) backward,
            // which keeps t_ij - x_ij s_ij from cancelling
            fw_record<AH>(A, P, ih, rec + slot * RS, arg, d2, dx, dy, dz, BACK ? d2 - fj : (SAVE ? d2 : fj), flag);
        };

        // lane = basis index: the walk over n records
        auto walk = [&](const int n) {
            const float4* R = reinterpret_cast<const float4*>(rec);
            for (int r = 0; r < n; r++, R += RS / 4) {
                const float4 u = R[0];
                const float fw = u.z;
                const int flag = __float_as_int(u.w);
                float u_back = 0.f;
                fw_gaussians<AH, false>(L, R, u, [&](const int k, const float g) {
                    if constexpr (BACK) u_back = fmaf(g, S[k], u_back);
                    else if constexpr (SAVE) { s[k] += g; T[k] = fmaf(g, fw, T[k]); }
                    else s[k] = fmaf(g, fw, s[k]);
                });
                if constexpr (BACK) { accB += u_back; accA = fmaf(u_back, fw, accA); }
                if (MODE != 0 && flag) flush(flag - 1);
            }
            if constexpr (MODE == 0) { pooled([&](const int k, const float v) { return v + s[k]; }); clear(); }
        };

        // a pair whose lattice range has no list: slab sweeps over (n1; n2, n3), lane = (n2, n3)
        auto sweep = [&](const int64_t e, auto&& body) {
            const float* Tc = A.tvecs + 9 * (int64_t)c;
            const float t1x = __ldg(Tc), t1y = __ldg(Tc + 1), t1z = __ldg(Tc + 2);
            const float t2x = __ldg(Tc + 3), t2y = __ldg(Tc + 4), t2z = __ldg(Tc + 5);
            const float t3x = __ldg(Tc + 6), t3y = __ldg(Tc + 7), t3z = __ldg(Tc + 8);
            const float rx = __ldg(A.pos_ij + 3 * e), ry = __ldg(A.pos_ij + 3 * e + 1), rz = __ldg(A.pos_ij + 3 * e + 2);
            const int L1 = 2 * R1 + 1, L3 = 2 * R3 + 1, L23 = (2 * R2 + 1) * L3;
            const float invL3 = 1.0f / (float)L3;
            const int nSub = (L23 + 31) >> 5;
            for (int sub = 0; sub < nSub; sub++) {
                const int idx = sub * 32 + lane;
                int q2 = (int)(((float)idx + 0.5f) * invL3), r3 = idx - q2 * L3;
                if (r3 < 0) { q2--; r3 += L3; } else if (r3 >= L3) { q2++; r3 -= L3; }
                const float n2 = ll_int_to_float(q2 - R2), n3 = ll_int_to_float(r3 - R3);
                const float ox = fmaf(t3x, n3, fmaf(t2x, n2, rx)), oy = fmaf(t3y, n3, fmaf(t2y, n2, ry)),
                            oz = fmaf(t3z, n3, fmaf(t2z, n2, rz));
                const bool valid = idx < L23;
                for (int k1 = 0; k1 < L1; k1++) {
                    const float n1 = ll_int_to_float(k1 - R1);
                    const float dx = fmaf(t1x, n1, ox), dy = fmaf(t1y, n1, oy), dz = fmaf(t1z, n1, oz);
                    body(valid, sub == nSub - 1 && k1 == L1 - 1, fmaf(dz, dz, fmaf(dy, dy, dx * dx)), dx, dy, dz);
                }
            }
        };

        // lane = (component, parity): V += sum over the tile's pairs of weight x rows[key atom]
        auto pool = [&](const float* src, const float weight, const int nt) {
            const float* vp = src + ((int64_t)(j0 + tile0) * H + h) * kAtHd + (lane & 15);
#pragma unroll 4
            for (int b = 0; b < nt; b += 2) {
                const int jj = b + (lane >> 4);
                const float w = __shfl_sync(0xffffffffu, weight, jj & 31);
                if (jj < nt) V = fmaf(w, __ldg(vp + (int64_t)jj * H * kAtHd), V);
            }
        };

        for (tile0 = 0; tile0 < np; tile0 += 32) {
            const int nt = min(32, np - tile0);
            const bool on = lane < nt;
            const int64_t e = e0 + tile0 + lane, j = (int64_t)j0 + tile0 + lane;
            // ---- lane = pair: q.k, normaliser, bias, soft-max weight ----
            float qk = 0.f, gov = 0.f;
            if (on) {
                if (__ldg(A.edges + A.E + e) != j) atomicOr(&g_status, CFB200_ST_PAIR_LAYOUT);       // not the dense layout
                const float* qp = A.qs + ih * kAtHd;
                const float* kp = A.k + (j * H + h) * kAtHd;
                if (A.vec) {
#pragma unroll
                    for (int d = 0; d < kAtHd / 4; d++) {
                        const float4 u = __ldg(reinterpret_cast<const float4*>(qp) + d), v = __ldg(reinterpret_cast<const float4*>(kp) + d);
                        qk = fmaf(u.x, v.x, fmaf(u.y, v.y, fmaf(u.z, v.z, fmaf(u.w, v.w, qk))));
                    }
                } else {
                    for (int d = 0; d < kAtHd; d++) qk = fmaf(__ldg(qp + d), __ldg(kp + d), qk);
                }
                if constexpr (BACK) {
                    const float* gp = A.gout + ih * kAtHd;
                    const float* vp = A.v + (j * H + h) * kAtHd;
                    if (A.vec) {
#pragma unroll
                        for (int d = 0; d < kAtHd / 4; d++) {
                            const float4 u = __ldg(reinterpret_cast<const float4*>(gp) + d), v = __ldg(reinterpret_cast<const float4*>(vp) + d);
                            gov = fmaf(u.x, v.x, fmaf(u.y, v.y, fmaf(u.z, v.z, fmaf(u.w, v.w, gov))));
                        }
                    } else {
                        for (int d = 0; d < kAtHd; d++) gov = fmaf(__ldg(gp + d), __ldg(vp + d), gov);
                    }
                }
            }
            float sum = 0.f, px = 0.f, ref = 0.f;
            float sum_lost = 0.f, px_lost = 0.f;            // what the additions below rounded away
            int cnt = 0;
            if (use_list) {
                const float* Lq = A.list + (size_t)(on ? e : e0) * kListStride;
                auto quad = [&](const int q) {
                    if (A.vec_list) return __ldg(reinterpret_cast<const float4*>(Lq) + q);
                    return make_float4(__ldg(Lq + 4 * q), __ldg(Lq + 4 * q + 1), __ldg(Lq + 4 * q + 2), __ldg(Lq + 4 * q + 3));
                };
                float4 u = quad(0);
                ref = u.x;
                for (int q = 0; q < kListLen / 4; q++) {
                    const float4 v = u;
                    if (q + 1 < kListLen / 4) u = quad(q + 1);
                    const float d4[4] = {v.x, v.y, v.z, v.w};
                    float arg = 0.f, w4[4], x4[4];
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        arg = a * (d4[x] - ref);
                        w4[x] = arg > -cut ? ex2_approx(arg * kLlLog2e) : 0.f;
                        x4[x] = arg > -cut ? (BACK ? d4[x] - ref : d4[x]) : 0.f;
                        cnt += arg > -P.prune ? 1 : 0;
                    }
                    // Up to 125 weights in one chain would round two to five times as much as one per lane and a tree.  So
                    // four at a time, and what an addition loses is kept: sorted weights make the sum the larger operand.
                    // Error of a pair's mean d^2 against 64 bits (mean square; cells of 2.5-10 / 1.2-5 A): one chain 2.1 /
                    // 3.3e-7, tree over the lanes 8.7 / 7.1e-8, this 7.8 / 5.9e-8, for 1.2 % of a training step.
                    const float qs = (w4[0] + w4[1]) + (w4[2] + w4[3]), ts = sum + qs;
                    sum_lost += qs - (ts - sum);
                    sum = ts;
                    if (MODE != 0) {
                        const float qx = fmaf(w4[0], x4[0], w4[1] * x4[1]) + fmaf(w4[2], x4[2], w4[3] * x4[3]), tx = px + qx;
                        px_lost += qx - (tx - px);
                        px = tx;
                    }
                    if (!__any_sync(0xffffffffu, arg > -cut)) break;     // sorted: nothing behind it counts
                }
                // the nearest translation always counts (a coefficient that is not a number compares false everywhere)
                cnt = on ? max(cnt, 1) : 0;
                if (!(a == a)) sum = a;
                if (sum_lost == sum_lost) sum += sum_lost;  // (an infinite sum has lost nothing)
                if (px_lost == px_lost) px += px_lost;
            } else {
                // Backward: weights come from the pair's bias, so the sweep that makes the records is the only one, and d^2
                // counts from z / a, at most log(125) / |a| from the nearest one's.  (A training step of eight cells of 100-200
                // atoms without lists: 14.4 ms with a sweep for the distance and one for the normaliser before it, 12.2 without.)
                if constexpr (BACK) {
                    const float zv = on ? __ldg(A.z_in + e * H + h) : 0.f;
                    ref = fabsf(a) > 1e-20f ? zv / a : 0.f;
                    sum = __expf(fmaf(-a, ref, zv));        // 1 but for the quotient's rounding
                } else {
                    for (int jj = 0; jj < nt; jj++) {
                        float d2min = 1e10f, sl = 0.f, pl = 0.f;
                        sweep(e0 + tile0 + jj, [&](const bool valid, bool, const float d2, float, float, float) {
                            if (valid) d2min = fminf(d2min, d2);
                        });
                        d2min = warp_min(d2min);
                        sweep(e0 + tile0 + jj, [&](const bool valid, bool, const float d2, float, float, float) {
                            if (valid) {
                                const float w = ex2_approx(a * (d2 - d2min) * kLlLog2e);
                                sl += w;
                                pl = fmaf(w, d2, pl);
                            }
                        });
                        sl = warp_sum(sl);
                        if (SAVE) pl = warp_sum(pl);
                        if (lane == jj) { sum = sl; px = pl; ref = d2min; }
                    }
                }
            }
            inv = 1.0f / sum;
            float p = 0.f;
            if constexpr (BACK) {
                p = on ? __expf(qk + __ldg(A.z_in + e * H + h) - lse) : 0.f;
            } else {
                const float zv = logf(sum) + ref * a;
                if (on) {
                    A.z[e * H + h] = zv;
                    if (SAVE) A.px[e * H + h] = px * inv;
                }
                const float sj = qk + zv;
                float mt = on ? sj : -INFINITY;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
                mt = fmaxf(m, mt);
                p = on ? __expf(sj - mt) : 0.f;
                f = on ? p * inv : 0.f;
                if (tile0 > 0) {
                    const float sc = __expf(m - mt);
                    l *= sc; V *= sc;
#pragma unroll
                    for (int r = 0; r < NS; r++) { S[r] *= sc; if constexpr (SAVE) Tq[r] *= sc; }
                    if constexpr (MODE == 0) pooled([&](const int, const float v) { return v * sc; });
                }
                m = mt;
                l += p;
                pool(A.v, p, nt);
            }
            // ---- translations ----
            const bool faint = MODE != 1 && p < kFwFaint;       // a weight that is not a number is walked
            if (BACK) cA = cB = 0.f;
            if (use_list) {
                if (faint) cnt = 0;
                int pre = cnt;                              // inclusive, then exclusive prefix over the tile's pairs
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, pre, o); if (lane >= o) pre += u; }
                const int total = __shfl_sync(0xffffffffu, pre, 31);
                pre -= cnt;
                for (int f0 = 0; f0 < total; f0 += 32) {
                    const int idx = f0 + lane;
                    int jj = 0;                             // the pair translation idx belongs to: the last with pre <= idx
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const int u = __shfl_sync(0xffffffffu, pre, jj + o);
                        if (u <= idx) jj += o;
                    }
                    jj = min(jj, nt - 1);
                    const int k = idx - __shfl_sync(0xffffffffu, pre, jj), cj = __shfl_sync(0xffffffffu, cnt, jj);
                    const float rj = __shfl_sync(0xffffffffu, ref, jj), fj = BACK ? rj : __shfl_sync(0xffffffffu, f, jj);
                    if (idx < total) {
                        const float* Lp = A.list + (size_t)(e0 + tile0 + jj) * kListStride + k;
                        const float d2 = __ldg(Lp);
                        make_record(lane, a * (d2 - rj), d2, __ldg(Lp + kListLen), __ldg(Lp + 2 * kListLen), __ldg(Lp + 3 * kListLen),
                                    fj, k == cj - 1 ? jj + 1 : 0);
                    }
                    __syncwarp();
                    walk(min(32, total - f0));
                    __syncwarp();
                }
            } else {
                for (int jj = 0; jj < nt; jj++) {
                    if (__shfl_sync(0xffffffffu, faint ? 1 : 0, jj)) continue;
                    const float rj = __shfl_sync(0xffffffffu, ref, jj), fj = BACK ? rj : __shfl_sync(0xffffffffu, f, jj);
                    // survivors gather in the stage; records are made when 32 wait, and for the rest at the end
                    int waiting = 0;
                    auto emit = [&]() {
                        const int n = min(waiting, 32);
                        if (lane < n)
                            make_record(lane, stage[lane], stage[kFwStage + lane], stage[2 * kFwStage + lane], stage[3 * kFwStage + lane],
                                        stage[4 * kFwStage + lane], fj, 0);
                        __syncwarp();
                        walk(n);
                        waiting -= n;
                        float keep[5];
#pragma unroll
                        for (int x = 0; x < 5; x++) keep[x] = stage[x * kFwStage + 32 + lane];
                        __syncwarp();
#pragma unroll
                        for (int x = 0; x < 5; x++) stage[x * kFwStage + lane] = keep[x];
                        __syncwarp();
                    };
                    float pl = 0.f;                         // backward: this lane's part of sum w (d^2 - ref)
                    sweep(e0 + tile0 + jj, [&](const bool valid, const bool last, const float d2, const float dx, const float dy, const float dz) {
                        const float arg = a * (d2 - rj);
                        if (BACK && valid) pl = fmaf(ex2_approx(arg * kLlLog2e), d2 - rj, pl);
                        const bool keep = valid && arg > -(BACK ? P.prune + kFwLogBox : P.prune);
                        const unsigned mask = __ballot_sync(0xffffffffu, keep);
                        if (keep) {
                            float* o = stage + waiting + __popc(mask & ((1u << lane) - 1));
                            o[0] = arg; o[kFwStage] = d2; o[2 * kFwStage] = dx; o[3 * kFwStage] = dy; o[4 * kFwStage] = dz;
                        }
                        waiting += __popc(mask);
                        __syncwarp();
                        while (waiting >= 32 || (last && waiting > 0)) emit();
                    });
                    if constexpr (BACK) {
                        pl = warp_sum(pl);
                        if (lane == jj) px = pl;
                    }
                    if (MODE != 0) flush(jj);
                }
            }
            if constexpr (BACK) {
                if (waiting_pairs > 0) drain();
                // gradient with respect to the bias: p (gout . (v_j + W s_ij) - gout . out_i); coefficient gradient:
                //   c_dist x gz + p gout . W (t_ij - x s_ij)
                // (the reference scales the whole length-kernel result, gz term included, by the distance coefficient,
                // models/cuda_funcs/real_space_framed_proj.py:183)
                const float x = px * inv, B = cB * inv;        // x, and t_ij behind cA, count d^2 from the nearest one's
                const float gz = on ? p * (gov + B - D) : 0.f;
                if (on) {
                    A.gz[e * H + h] = gz;
                    ga += fmaf(P.c_dist * (x + ref), gz, p * (cA * inv - x * B));
                }
                pool(A.k, gz, nt);
            }
        }
        // an atom's results go to its row, a chunk's to a partial row (numbered from N)
        const bool partial = TASKS && row >= (int)A.N;
        const int64_t rh = (int64_t)(partial ? row - (int)A.N : row) * H + h;
        V += __shfl_xor_sync(0xffffffffu, V, 16);
        if constexpr (BACK) {
            ga = warp_sum(ga);
            if (lane == 0) (partial ? A.part_ga : A.ga)[rh] = ga;
            if (lane < kAtHd) (partial ? A.part_gq : A.gq)[rh * kAtHd + lane] = V;
            continue;
        }
        if constexpr (MODE == 0) pooled([&](const int k, const float v) { return S[k] = v; });
        l = warp_sum(l);
        const float inv_l = np > 0 ? 1.0f / l : 0.f;
        if (lane == 0) (partial ? A.part_lse : A.lse)[rh] = m + logf(l);
        // pooled basis sums: to memory with the scaling of the weight gradients, to shared memory for the projection
        float* sp = (partial ? A.part_spool : A.spool) + rh * kAtK;
#pragma unroll
        for (int r = 0; r < NS; r++) { S[r] *= inv_l; if constexpr (SAVE) Tq[r] *= inv_l; }
        sp[lane] = S[0]; sp[32 + lane] = S[1];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            sp[64 + 64 * x + lane] = AH > 0 ? S[AH > 0 ? 2 + AH * x : 0] * P.c_ang : 0.f;
            sp[96 + 64 * x + lane] = AH > 1 ? S[AH > 1 ? 3 + AH * x : 0] * P.c_ang : 0.f;
        }
#pragma unroll
        for (int r = 0; r < (SAVE ? 2 : 1); r++) {
            float* w = rows + r * K;
            const float* src = r == 0 ? S : Tq;
            *reinterpret_cast<float2*>(w + 2 * lane) = make_float2(src[0], src[1]);
            if constexpr (AH == 2) {
#pragma unroll
                for (int x = 0; x < 3; x++) *reinterpret_cast<float2*>(w + 64 + 64 * x + 2 * lane) = make_float2(src[2 + 2 * x], src[3 + 2 * x]);
            } else if constexpr (AH == 1) {
#pragma unroll
                for (int x = 0; x < 3; x++) w[64 + 32 * x + lane] = src[2 + x];
            }
        }
        __syncwarp();
        // out = (sum_j p_ij v_j + W S) / l; training: upool = W T / l
        V *= inv_l;
        const float2 o = fw_project<AH, SAVE ? 2 : 1>(W_s, rows, lane);
        const int d0 = fw_out(lane);
        const float v0 = __shfl_sync(0xffffffffu, V, d0), v1 = __shfl_sync(0xffffffffu, V, d0 + 1);
        if (fw_row(lane) == 0) {
            float* dst = (partial ? A.part_out : A.out) + rh * kAtHd + d0;
            dst[0] = v0 + o.x; dst[1] = v1 + o.y;
        }
        if (SAVE && fw_row(lane) == 1) {
            float* dst = (partial ? A.part_upool : A.upool) + rh * kAtHd + d0;
            dst[0] = o.x; dst[1] = o.y;
        }
        __syncwarp();
    }
    }   // heads in turn
}

// ---- the forward one pair after the other -------------------------------------------------------------------------
// Warp = (atom, head), its pairs in order, lane = basis index throughout (LatticeLane), each pair's 16 x 256 projection by
// itself, an online soft-max over the pairs; leaves per-pair results; sweeps each pair's translations.  Same results as
// attn_tile_kernel to rounding.  Bound by instruction issue.  Two uses:
// * batches without translation lists, where the tiles are no faster (see attn_fused_fwd);
// * tasks without a list in the training forward of models with weighted-PCA frames, whose order of summation is this one for
//   its rounding (attn_ordered_kernel forms the same sums in tiles from the lists; a training step of 16 crystals of 100-200
//   atoms 16.8 ms one pair after the other, 12.4 with that kernel, 8.2 with attn_tile_kernel).  An eigenvector of the second
//   moments has a sign and, where eigenvalues are close, a direction that a last bit decides, and the ReLUs behind it turn with
//   it.  In a batch whose errors have balanced signs the mean gradient is small, and one turned ReLU is then a quarter of its
//   root mean square: of 150 batches of 16 such crystals two moved by more than a tenth when the tiles' order of summation took
//   the place of this one, while the frames of the first layer, which come before it, stayed equal to the bit.  There the order
//   is part of the result.
constexpr int kPwStride = 260;         // W [16][260]: conflict-free 128-bit reads by 16 rows

// per-(atom, head) inputs
struct AtomTask {
    int64_t i, c, e0, e1;
    int R1, R2, R3;
};

template <bool ANG>
__device__ __forceinline__ AtomTask load_atom(const AtArgs& A, const Params& P, LatticeLane<2, ANG>& L, const int64_t i,
                                              const int h, const int lane)
{
    AtomTask T;
    const int H = P.H;
    T.i = i; T.c = A.batch[i];
    T.e0 = A.e_start[i]; T.e1 = A.e_start[i + 1];
    L.a = __ldg(A.a_ik + i * H + h);
    if constexpr (ANG) {
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const float* f = A.frame[x] + (i * H + h) * 3;
            L.fx[x] = __ldg(f); L.fy[x] = __ldg(f + 1); L.fz[x] = __ldg(f + 2);
        }
    }
    int Rl = 0;
    if (lane < 3) Rl = lattice_range_1d(P, L.a, P.cutoff_radius != 0.0f ? __ldg(A.rvlen + 3 * T.c + lane) : 0.0f);
    T.R1 = __shfl_sync(0xffffffffu, Rl, 0); T.R2 = __shfl_sync(0xffffffffu, Rl, 1); T.R3 = __shfl_sync(0xffffffffu, Rl, 2);
    return T;
}

constexpr int kPwWarps = 12;
constexpr size_t kPwSmem = sizeof(float) * (kAtHd * kPwStride + kPwWarps * 8 * 32 + kPwWarps * 3 * kAtK);

// out_d = W_d . row: lane = (output d, half of the 256 basis indices); every lane returns the full sum of its d.
// Packed FP32: two products per instruction, two partial sums.
// LD: floats between rows of W; GAP: floats between the halves of a row, of W and of the vector.
template <int LD, int GAP>
__device__ __forceinline__ float project_row(const float* W_s, const float* row, const int lane)
{
    const int d = lane & 15, half = lane >> 4;
    const ulonglong2* wr = reinterpret_cast<const ulonglong2*>(W_s + d * LD) + half * (32 + GAP / 4);
    const ulonglong2* sr = reinterpret_cast<const ulonglong2*>(row) + half * (32 + GAP / 4);
    f32x2 acc = pack2(0.f, 0.f);
#pragma unroll 8
    for (int k4 = 0; k4 < 32; k4++) {
        const ulonglong2 w4 = wr[k4], s4 = sr[k4];
        acc = fma2(s4.x, w4.x, acc);
        acc = fma2(s4.y, w4.y, acc);
    }
    float a0, a1;
    unpack2(acc, a0, a1);
    const float sum = a0 + a1;
    return sum + __shfl_xor_sync(0xffffffffu, sum, 16);
}

// One task, its pairs one after the other.  srow: 3 x 256 + GAP floats of the warp's (the basis vector being projected, the pooled
// sums plain and d^2-weighted); results go to row `row` (numbered from N: partial rows).
template <bool ANG, int LD, int GAP>
__device__ __forceinline__ void pairwise_task(const AtArgs& A, const Params& P, LatticeLane<2, ANG>& L, const AtomTask& T, int64_t row,
                                              const bool partial, const int h, const float* W_s, float* srow, const int lane)
{
    const int H = P.H;
    const int64_t i = T.i;
    // pooled basis sums of this lane as four packed pairs (indices l, l + 32 of each basis): Sp[32 x], x < 4; then the
    // d^2-weighted ones
    f32x2* Sp = reinterpret_cast<f32x2*>(srow + kAtK + GAP) + lane;
    f32x2* Tq = Sp + kAtK / 2;
    const float qd = lane < kAtHd ? __ldg(A.qs + (i * H + h) * kAtHd + lane) : 0.f;
    float m = -INFINITY, l = 0.f, V = 0.f;
#pragma unroll
    for (int x = 0; x < 4; x++) Sp[32 * x] = Tq[32 * x] = pack2(0.f, 0.f);        // attention-pooled sums, plain and d^2-weighted
    const int64_t j0 = T.e1 > T.e0 ? A.edges[A.E + T.e0] : 0;
    for (int64_t e = T.e0; e < T.e1; e++) {
        const int64_t j = j0 + (e - T.e0);
        if (lane == 0 && __ldg(A.edges + A.E + e) != j) atomicOr(&g_status, CFB200_ST_PAIR_LAYOUT);   // not the dense layout
        float kd = 0.f, vd = 0.f;
        if (lane < kAtHd) { kd = __ldg(A.k + (j * H + h) * kAtHd + lane); vd = __ldg(A.v + (j * H + h) * kAtHd + lane); }
        L.reset();
        L.run_slabs(P, T.R1, T.R2, T.R3, __ldg(A.pos_ij + 3 * e), __ldg(A.pos_ij + 3 * e + 1), __ldg(A.pos_ij + 3 * e + 2),
                    A.tvecs + 9 * T.c);
        float r0 = L.sum_l, r1 = L.px_l, r2 = qd * kd;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r0 += __shfl_xor_sync(0xffffffffu, r0, o); r1 += __shfl_xor_sync(0xffffffffu, r1, o);
            r2 += __shfl_xor_sync(0xffffffffu, r2, o);
        }
        const float sum = r0, qk = r2;
        const float inv = 1.0f / sum;
        const float zv = logf(sum) + L.ref * L.a;
        if (lane == 0) { A.z[e * H + h] = zv; A.px[e * H + h] = r1 * inv; }
        // the pair's value encoding: its normalised basis sums, with the scaling of the values, times W
        {
            const float cd = inv * P.c_dist, ca = inv * P.c_ang;
            srow[lane] = L.sd[0] * cd; srow[32 + lane] = L.sd[1] * cd;
#pragma unroll
            for (int x = 0; x < 3; x++) { srow[64 + 64 * x + (x > 0 ? GAP : 0) + lane] = L.sa[x][0] * ca; srow[96 + 64 * x + (x > 0 ? GAP : 0) + lane] = L.sa[x][1] * ca; }
        }
        __syncwarp();
        const float val_d = project_row<LD, GAP>(W_s, srow, lane);
        if (lane < kAtHd) A.val[(e * H + h) * kAtHd + lane] = val_d;
        __syncwarp();
        const float s = qk + zv;
        const float mn = fmaxf(m, s);
        const float sc = __expf(m - mn), p = __expf(s - mn);
        const float f = p * inv;
        l = fmaf(l, sc, p);
        V = fmaf(V, sc, p * (vd + val_d));
        {
            const f32x2 sc2 = pack2(sc, sc), f2 = pack2(f, f);
            Sp[0] = fma2(Sp[0], sc2, mul2(f2, pack2(L.sd[0], L.sd[1])));
            Tq[0] = fma2(Tq[0], sc2, mul2(f2, pack2(L.qd[0], L.qd[1])));
#pragma unroll
            for (int x = 0; x < 3; x++) {
                Sp[32 + 32 * x] = fma2(Sp[32 + 32 * x], sc2, mul2(f2, pack2(L.sa[x][0], L.sa[x][1])));
                Tq[32 + 32 * x] = fma2(Tq[32 + 32 * x], sc2, mul2(f2, pack2(L.qa[x][0], L.qa[x][1])));
            }
        }
        m = mn;
    }
    const float inv_l = T.e1 > T.e0 ? 1.0f / l : 0.f;
    if (partial) row -= A.N;
    if (lane == 0) (partial ? A.part_lse : A.lse)[row * H + h] = m + logf(l);
    float* sp = (partial ? A.part_spool : A.spool) + (row * H + h) * kAtK;
    {
        float s0, s1, t0, t1;
        unpack2(Sp[0], s0, s1); unpack2(Tq[0], t0, t1);
        sp[lane] = s0 * inv_l; sp[32 + lane] = s1 * inv_l;
        srow[lane] = t0 * inv_l * P.c_dist; srow[32 + lane] = t1 * inv_l * P.c_dist;
#pragma unroll
        for (int x = 0; x < 3; x++) {
            unpack2(Sp[32 + 32 * x], s0, s1); unpack2(Tq[32 + 32 * x], t0, t1);
            sp[64 + 64 * x + lane] = s0 * inv_l * P.c_ang; sp[96 + 64 * x + lane] = s1 * inv_l * P.c_ang;
            srow[64 + 64 * x + (x > 0 ? GAP : 0) + lane] = t0 * inv_l * P.c_ang; srow[96 + 64 * x + (x > 0 ? GAP : 0) + lane] = t1 * inv_l * P.c_ang;
        }
    }
    __syncwarp();
    const float up_d = project_row<LD, GAP>(W_s, srow, lane);     // W (pooled d^2-weighted sums)
    if (lane < kAtHd) {
        (partial ? A.part_out : A.out)[(row * H + h) * kAtHd + lane] = V * inv_l;
        (partial ? A.part_upool : A.upool)[(row * H + h) * kAtHd + lane] = up_d;
    }
    __syncwarp();
}

template <bool ANG, bool TASKS>
__global__ void __launch_bounds__(kPwWarps * 32, 2) attn_pairwise_kernel(const AtArgs A, const Params P)
{
    wait_for_predecessors();
    extern __shared__ __align__(16) float smem[];
    float* W_s = smem;                                      // [16][260]
    float* tbuf = W_s + kAtHd * kPwStride;                  // per warp 8 x 32
    float* rows = tbuf + kPwWarps * 8 * 32;                 // per warp 256: the basis vector being projected
    const int H = P.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    LatticeLane<2, ANG> L;
    L.init(P, lane, tbuf + warp * 8 * 32);
    float* srow = rows + warp * 3 * kAtK;
    __shared__ int head_open;

    // heads in turn, as in attn_tile_kernel
    for (int turn = 0; turn < 2 * H; turn++) {
    int h = blockIdx.y;
    if (turn > 0) {
        __syncthreads();                                    // every warp is done with the previous head's weights
        if (threadIdx.x == 0) {
            // the head with the most entries left in its queue (a stale count costs a wasted or a missed turn at most)
            int best = -1, most = 0;
            for (int hh = 0; hh < H; hh++) {
                const int limit = TASKS ? (int)(A.n_entries - kSplitSlots) + __ldg(A.chunk_count + hh) : (int)A.N;
                const int left = limit - atomicAdd(A.counters + hh, 0);
                if (left > most) { most = left; best = hh; }
            }
            head_open = best;
        }
        __syncthreads();
        h = head_open;
        if (h < 0) break;                                   // every queue is drained
    }
    const int first = TASKS ? kSplitSlots - __ldg(A.chunk_count + h) : 0;
    for (int idx = threadIdx.x; idx < kAtHd * kAtK / 4; idx += kPwWarps * 32) {
        const int o = idx >> 6, k4 = idx & 63, b = k4 >> 4, d4 = k4 & 15;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        const int width = b == 0 ? 64 : P.angle_dim;          // columns this basis' weights hold (zero beyond)
        if (A.W[b] != nullptr && 4 * d4 < width) {
            const float* src = A.W[b] + ((size_t)h * kAtHd + o) * width + 4 * d4;
            w = make_float4(__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3));
        }
        reinterpret_cast<float4*>(W_s)[o * (kPwStride / 4) + k4] = w;
    }
    __syncthreads();

    for (;;) {
        const int64_t t = next_task(A.counters + h, lane) + first;
        if (t >= (TASKS ? A.n_entries : A.N)) break;
        int64_t i, row;
        AtomTask T;
        if (TASKS) {
            const int4 d = __ldg(A.tasks + (size_t)h * A.n_entries + t);
            const int cnt = d.w & 0xFFFFFF;
            if (cnt == 0) continue;
            i = d.x; row = d.y;
            T = load_atom(A, P, L, i, h, lane);
            T.e0 += d.z; T.e1 = T.e0 + cnt;
        } else {
            i = A.order != nullptr ? (int64_t)A.order[t] : t;
            row = i;
            T = load_atom(A, P, L, i, h, lane);
        }
        pairwise_task<ANG, kPwStride, 0>(A, P, L, T, row, TASKS && row >= A.N, h, W_s, srow, lane);
    }
    }   // heads in turn
}

// ---- the same sums in tiles ---------------------------------------------------------------------------------------
// The forward one pair after the other, for tasks whose ranges have lists, with lanes used as in attn_tile_kernel and every
// sum formed in the order of pairwise_task, so that each result is the same to the bit:
//   * normaliser and mean d^2: lane = translation, four of the 125 per lane, then the tree of a butterfly over the lanes --
//     walked for eight pairs at once, lane = (pair, quarter of the tree's leaves);
//   * lane = pair: q.k as the butterfly adds its 16 products, logarithm, bias; the running maximum is a prefix maximum, and
//     with it every factor of the online soft-max is known before the walk;
//   * lane = translation: records; lane = basis index: the walk, which meets a pair's translations in the same order;
//   * projection of four pairs at once: a lane runs the chains of two outputs and two pairs over half of the indices.
// Bound by shared memory (the projection's reads: 133 wavefronts per pair and head, 60 % of the data path; 1.82 ms before its
// rows were kept in different banks) and issue (490 instructions instead of 803, 55 % of the slots).  16 crystals of 100-200
// atoms (2.7 M pairs and heads), per launch 2.65 -> 1.70 ms; a training step 16.8 -> 12.4 ms.
constexpr int kOrWarps = 10;
constexpr int kOrWait = 36;            // stride of the waiting partial sums: conflict-free 64-bit reads by (pair, quarter)
// A row is two halves 16 banks apart, and two rows are 8 banks apart: the four addresses that a warp reads a row or W at meet
// in as few banks as they can.
constexpr int kOrGap = 16, kOrRow = 2 * 128 + kOrGap + 4;
constexpr int kOrWarpFloats = 4 * kOrRow + 32 * kFwRec + 8 * kOrWait * 2 + 32 * 4;
constexpr size_t kOrSmem = sizeof(float) * (kAtHd * kOrRow + kOrWarps * kOrWarpFloats);

// tasks whose ranges have no list; not inlined, so that its registers are not the kernel's
template <bool TASKS>
__device__ __noinline__ void ordered_slow_task(const AtArgs& A, const Params& P, const int i, const int off, const int np, const int64_t row,
                                               const int h, const float* W_s, float* warp_s)
{
    const int lane = threadIdx.x & 31;
    LatticeLane<2, true> L;
    L.init(P, lane, warp_s + 3 * kAtK + kOrGap);
    AtomTask T = load_atom(A, P, L, i, h, lane);
    T.e0 += off; T.e1 = T.e0 + np;
    pairwise_task<true, kOrRow, kOrGap>(A, P, L, T, row, TASKS && row >= A.N, h, W_s, warp_s, lane);
}

template <bool TASKS>
__global__ void __launch_bounds__(kOrWarps * 32, 2) attn_ordered_kernel(const __grid_constant__ AtArgs A, const __grid_constant__ Params P)
{
    wait_for_predecessors();
    extern __shared__ __align__(16) float smem[];
    float* W_s = smem;                                      // [16][kOrRow]
    const int H = P.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* rows = W_s + kAtHd * kOrRow + warp * kOrWarpFloats;           // four basis vectors being projected
    float* rec = rows + 4 * kOrRow;
    float2* wait = reinterpret_cast<float2*>(rec + 32 * kFwRec);            // [8][kOrWait]: lanes' parts of normaliser and sum w d^2
    float4* pairs = reinterpret_cast<float4*>(rec + 32 * kFwRec + 8 * kOrWait * 2);    // per pair of the tile: sc, p, f, 1 / sum
    const FwLane L(P, lane);
    const bool vec = A.vec;
    __shared__ int head_open;

    // heads in turn, as in attn_tile_kernel
    for (int turn = 0; turn < 2 * H; turn++) {
    int h = blockIdx.y;
    if (turn > 0) {
        __syncthreads();                                    // every warp is done with the previous head's weights
        if (threadIdx.x == 0) {
            int best = -1, most = 0;
            for (int hh = 0; hh < H; hh++) {
                const int limit = TASKS ? (int)(A.n_entries - kSplitSlots) + __ldg(A.chunk_count + hh) : (int)A.N;
                const int left = limit - atomicAdd(A.counters + hh, 0);
                if (left > most) { most = left; best = hh; }
            }
            head_open = best;
        }
        __syncthreads();
        h = head_open;
        if (h < 0) break;                                   // every queue is drained
    }
    const int first = TASKS ? kSplitSlots - __ldg(A.chunk_count + h) : 0;
    for (int idx = threadIdx.x; idx < kAtHd * kAtK; idx += kOrWarps * 32) {
        const int o = idx >> 8, b = (idx >> 6) & 3, d = idx & 63;
        const int width = b == 0 ? 64 : P.angle_dim;        // columns this basis' weights hold (zero beyond)
        W_s[o * kOrRow + (idx & 255) + (b > 1 ? kOrGap : 0)] = d < width ? __ldg(A.W[b] + ((size_t)h * kAtHd + o) * width + d) : 0.f;
    }
    __syncthreads();

    for (;;) {
        const int64_t t = next_task(A.counters + h, lane) + first;
        if (t >= (TASKS ? A.n_entries : A.N)) break;
        int i, row, off = 0, np;
        int64_t e0;
        if (TASKS) {
            const int4 d = __ldg(A.tasks + (size_t)h * A.n_entries + t);
            np = d.w & 0xFFFFFF;
            if (np == 0) continue;
            i = d.x; row = d.y; off = d.z;
            e0 = A.e_start[i];
        } else {
            i = A.order != nullptr ? A.order[t] : (int)t;
            row = i;
            e0 = A.e_start[i];
            np = (int)(A.e_start[i + 1] - e0);
        }
        const int64_t ih = (int64_t)i * H + h;
        const float a = __ldg(A.a_ik + ih);
        int Rl = A.cache_range;
        if (lane < 3) Rl = lattice_range_1d(P, a, P.cutoff_radius != 0.0f ? __ldg(A.rvlen + 3 * A.batch[i] + lane) : 0.0f);
        if (__any_sync(0xffffffffu, Rl != A.cache_range)) {
            ordered_slow_task<TASKS>(A, P, i, off, np, row, h, W_s, rows);
            continue;
        }
        e0 += off;
        const int j0 = np > 0 ? (int)A.edges[A.E + e0] : 0;
        float m = -INFINITY, l = 0.f, V = 0.f;
        float s[8], T[8];                                   // the pair's sums, plain and d^2-weighted
        f32x2 S[4], Tq[4];                                  // both pooled
#pragma unroll
        for (int r = 0; r < 8; r++) s[r] = T[r] = 0.f;
#pragma unroll
        for (int x = 0; x < 4; x++) S[x] = Tq[x] = pack2(0.f, 0.f);
        int tile0 = 0;

        auto flush = [&](const int j) {
            const float4 pr = pairs[j];                     // sc, p, f, 1 / sum
            {
                const float cd = pr.w * P.c_dist, ca = pr.w * P.c_ang;
                float* w = rows + (j & 3) * kOrRow + lane;
                w[0] = s[0] * cd; w[32] = s[1] * cd;
#pragma unroll
                for (int x = 1; x < 4; x++) {
                    const int at = 64 * x + (x > 1 ? kOrGap : 0);
                    w[at] = s[2 * x] * ca; w[at + 32] = s[2 * x + 1] * ca;
                }
            }
            l = fmaf(l, pr.x, pr.y);
            const f32x2 sc2 = pack2(pr.x, pr.x), f2 = pack2(pr.z, pr.z);
#pragma unroll
            for (int x = 0; x < 4; x++) {
                S[x] = fma2(S[x], sc2, mul2(f2, pack2(s[2 * x], s[2 * x + 1])));
                Tq[x] = fma2(Tq[x], sc2, mul2(f2, pack2(T[2 * x], T[2 * x + 1])));
            }
#pragma unroll
            for (int r = 0; r < 8; r++) s[r] = T[r] = 0.f;
            if ((j & 3) != 3 && tile0 + j != np - 1) return;
            // value encodings of up to four pairs: lane = (half of the indices, pair of pairs, outputs o and o + 8)
            const int n = (j & 3) + 1, o = lane & 7, rp = (lane >> 3) & 1, half = lane >> 4;
            const int64_t ef = e0 + tile0 + (j & ~3);
            const float* vp = A.v + ((int64_t)(j0 + tile0 + (j & ~3)) * H + h) * kAtHd + (lane & 15);
            float vd[4];
#pragma unroll
            for (int r = 0; r < 4; r++) vd[r] = r < n ? __ldg(vp + (int64_t)r * H * kAtHd) : 0.f;
            __syncwarp();
            const ulonglong2* w0 = reinterpret_cast<const ulonglong2*>(W_s + o * kOrRow) + half * (32 + kOrGap / 4);
            const ulonglong2* w1 = w0 + 8 * kOrRow / 4;
            const ulonglong2* r0 = reinterpret_cast<const ulonglong2*>(rows + 2 * rp * kOrRow) + half * (32 + kOrGap / 4);
            const ulonglong2* r1 = r0 + kOrRow / 4;
            f32x2 acc[2][2];
            acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = pack2(0.f, 0.f);
#pragma unroll 4
            for (int k = 0; k < 32; k++) {
                const ulonglong2 wa = w0[k], wb = w1[k], ra = r0[k], rb = r1[k];
                acc[0][0] = fma2(ra.x, wa.x, acc[0][0]); acc[0][0] = fma2(ra.y, wa.y, acc[0][0]);
                acc[0][1] = fma2(ra.x, wb.x, acc[0][1]); acc[0][1] = fma2(ra.y, wb.y, acc[0][1]);
                acc[1][0] = fma2(rb.x, wa.x, acc[1][0]); acc[1][0] = fma2(rb.y, wa.y, acc[1][0]);
                acc[1][1] = fma2(rb.x, wb.x, acc[1][1]); acc[1][1] = fma2(rb.y, wb.y, acc[1][1]);
            }
            float q[2];                                     // this lane passes on output o + 8 half of its two pairs
#pragma unroll
            for (int r = 0; r < 2; r++) {
                float x, y, v[2];
                unpack2(acc[r][0], x, y);
                v[0] = x + y;
                unpack2(acc[r][1], x, y);
                v[1] = x + y;
#pragma unroll
                for (int c = 0; c < 2; c++) v[c] = v[c] + __shfl_xor_sync(0xffffffffu, v[c], 16);
                q[r] = half ? v[1] : v[0];
                if (2 * rp + r < n) A.val[((ef + 2 * rp + r) * H + h) * kAtHd + o + 8 * half] = q[r];
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float val_d = __shfl_sync(0xffffffffu, q[r & 1], ((lane & 8) << 1) + (r >> 1) * 8 + (lane & 7));
                if (r < n) {
                    const float4 pv = pairs[(j & ~3) + r];
                    V = fmaf(V, pv.x, pv.y * (vd[r] + val_d));
                }
            }
            __syncwarp();
        };

        for (tile0 = 0; tile0 < np; tile0 += 32) {
            const int nt = min(32, np - tile0);
            const bool on = lane < nt;
            const int64_t e = e0 + tile0 + lane, j = (int64_t)j0 + tile0 + lane;
            // ---- lane = translation: normalisers, eight pairs at a time ----
            float sum = 1.f, px = 0.f;
            int cnt = 0;
            for (int g = 0; g < nt; g += 8) {
                const int n = min(8, nt - g);
                const float* Ll = A.list + (size_t)(e0 + tile0 + g) * kListStride + lane;
#pragma unroll 4
                for (int k = 0; k < n; k++, Ll += kListStride) {
                    const float d0 = __ldg(Ll), d1 = __ldg(Ll + 32), d2 = __ldg(Ll + 64), d3 = __ldg(Ll + 96);
                    const float ref = __shfl_sync(0xffffffffu, d0, 0);
                    const float a0 = a * (d0 - ref), a1 = a * (d1 - ref), a2 = a * (d2 - ref), a3 = a * (d3 - ref);
                    const float w0 = ex2_approx(a0 * kLlLog2e), w1 = ex2_approx(a1 * kLlLog2e), w2 = ex2_approx(a2 * kLlLog2e),
                                w3 = ex2_approx(a3 * kLlLog2e);
                    wait[k * kOrWait + lane] = make_float2(((w0 + w1) + w2) + w3, fmaf(w3, d3, fmaf(w2, d2, fmaf(w1, d1, w0 * d0))));
                    int c = __popc(__ballot_sync(0xffffffffu, a0 > -P.prune));
                    if (c == 32) {
                        c += __popc(__ballot_sync(0xffffffffu, a1 > -P.prune));
                        if (c == 64) {
                            c += __popc(__ballot_sync(0xffffffffu, a2 > -P.prune));
                            c += __popc(__ballot_sync(0xffffffffu, a3 > -P.prune));
                        }
                    }
                    if (lane == g + k) cnt = c;
                }
                __syncwarp();
                // the butterfly adds lanes 16 apart, then 8, 4, 2, 1
                const float2* p = wait + (lane >> 2) * kOrWait + (lane & 3);
                float2 x[8];
#pragma unroll
                for (int k = 0; k < 8; k++) x[k] = p[4 * k];
                float r0 = ((x[0].x + x[4].x) + (x[2].x + x[6].x)) + ((x[1].x + x[5].x) + (x[3].x + x[7].x));
                float r1 = ((x[0].y + x[4].y) + (x[2].y + x[6].y)) + ((x[1].y + x[5].y) + (x[3].y + x[7].y));
                r0 += __shfl_xor_sync(0xffffffffu, r0, 2); r1 += __shfl_xor_sync(0xffffffffu, r1, 2);
                r0 += __shfl_xor_sync(0xffffffffu, r0, 1); r1 += __shfl_xor_sync(0xffffffffu, r1, 1);
                const int from = ((lane - g) & 7) * 4;
                r0 = __shfl_sync(0xffffffffu, r0, from); r1 = __shfl_sync(0xffffffffu, r1, from);
                if ((lane & ~7) == g) { sum = r0; px = r1; }
                __syncwarp();
            }
            // ---- lane = pair ----
            float ref = 0.f, qk = 0.f;
            if (on) {
                if (__ldg(A.edges + A.E + e) != j) atomicOr(&g_status, CFB200_ST_PAIR_LAYOUT);       // not the dense layout
                ref = __ldg(A.list + (size_t)e * kListStride);
                const float* qp = A.qs + ih * kAtHd;
                const float* kp = A.k + (j * H + h) * kAtHd;
                float x[kAtHd];
                if (vec) {
#pragma unroll
                    for (int d = 0; d < kAtHd / 4; d++) {
                        const float4 u = __ldg(reinterpret_cast<const float4*>(qp) + d), v = __ldg(reinterpret_cast<const float4*>(kp) + d);
                        x[4 * d] = __fmul_rn(u.x, v.x); x[4 * d + 1] = __fmul_rn(u.y, v.y);
                        x[4 * d + 2] = __fmul_rn(u.z, v.z); x[4 * d + 3] = __fmul_rn(u.w, v.w);
                    }
                } else {
#pragma unroll
                    for (int d = 0; d < kAtHd; d++) x[d] = __fmul_rn(__ldg(qp + d), __ldg(kp + d));
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                    for (int d = 0; d < o; d++) x[d] = __fadd_rn(x[d], x[d + o]);
                qk = x[0];
                cnt = max(cnt, 1);          // the nearest translation always counts (a coefficient that is not a number)
            }
            const float inv = 1.0f / sum;
            const float zv = logf(sum) + ref * a;
            const float sj = qk + zv;
            float mx = on ? sj : -INFINITY;                 // running maximum up to this pair
            if (lane == 0) mx = fmaxf(m, mx);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, mx, o); if (lane >= o) mx = fmaxf(u, mx); }
            float before = __shfl_up_sync(0xffffffffu, mx, 1);
            if (lane == 0) before = m;
            const float sc = __expf(before - mx), p = __expf(sj - mx);
            m = __shfl_sync(0xffffffffu, mx, 31);
            if (on) {
                A.z[e * H + h] = zv;
                A.px[e * H + h] = px * inv;
                pairs[lane] = make_float4(sc, p, p * inv, inv);
            }
            // ---- translations, as in attn_tile_kernel ----
            int pre = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, pre, o); if (lane >= o) pre += u; }
            const int total = __shfl_sync(0xffffffffu, pre, 31);
            pre -= cnt;
            for (int f0 = 0; f0 < total; f0 += 32) {
                const int idx = f0 + lane;
                int jj = 0;                                 // the pair translation idx belongs to: the last with pre <= idx
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const int u = __shfl_sync(0xffffffffu, pre, jj + o);
                    if (u <= idx) jj += o;
                }
                jj = min(jj, nt - 1);
                const int k = idx - __shfl_sync(0xffffffffu, pre, jj), cj = __shfl_sync(0xffffffffu, cnt, jj);
                const float rj = __shfl_sync(0xffffffffu, ref, jj);
                if (idx < total) {
                    const float* Lp = A.list + (size_t)(e0 + tile0 + jj) * kListStride + k;
                    const float d2 = __ldg(Lp);
                    fw_record<2>(A, P, ih, rec + lane * kFwRec, a * (d2 - rj), d2, __ldg(Lp + kListLen), __ldg(Lp + 2 * kListLen),
                                 __ldg(Lp + 3 * kListLen), d2, k == cj - 1 ? jj + 1 : 0);
                }
                __syncwarp();
                const float4* R = reinterpret_cast<const float4*>(rec);
                const int n = min(32, total - f0);
                for (int r = 0; r < n; r++, R += kFwRec / 4) {
                    const float4 u = R[0];
                    const float d2 = u.z;
                    const int flag = __float_as_int(u.w);
                    fw_gaussians<2, true>(L, R, u, [&](const int x, const float g) { s[x] += g; T[x] = fmaf(g, d2, T[x]); });
                    if (flag) flush(flag - 1);
                }
                __syncwarp();
            }
        }
        const float inv_l = np > 0 ? 1.0f / l : 0.f;
        const bool partial = TASKS && row >= (int)A.N;
        const int64_t rh = (int64_t)(partial ? row - (int)A.N : row) * H + h;
        if (lane == 0) (partial ? A.part_lse : A.lse)[rh] = m + logf(l);
        float* sp = (partial ? A.part_spool : A.spool) + rh * kAtK + lane;
#pragma unroll
        for (int x = 0; x < 4; x++) {
            float s0, s1, t0, t1;
            unpack2(S[x], s0, s1); unpack2(Tq[x], t0, t1);
            if (x == 0) {
                sp[0] = s0 * inv_l; sp[32] = s1 * inv_l;
                rows[lane] = t0 * inv_l * P.c_dist; rows[32 + lane] = t1 * inv_l * P.c_dist;
            } else {
                sp[64 * x] = s0 * inv_l * P.c_ang; sp[64 * x + 32] = s1 * inv_l * P.c_ang;
                float* w = rows + 64 * x + (x > 1 ? kOrGap : 0) + lane;
                w[0] = t0 * inv_l * P.c_ang; w[32] = t1 * inv_l * P.c_ang;
            }
        }
        __syncwarp();
        const float up_d = project_row<kOrRow, kOrGap>(W_s, rows, lane);     // W (pooled d^2-weighted sums)
        if (lane < kAtHd) {
            (partial ? A.part_out : A.out)[rh * kAtHd + lane] = V * inv_l;
            (partial ? A.part_upool : A.upool)[rh * kAtHd + lane] = up_d;
        }
        __syncwarp();
    }
    }   // heads in turn
}

// Backward pass from the results of the training forward.  Per pair
//   p = exp(q.k + z - lse),  gz = p (gout . (v_j + values_ij) - gout . out_i),
//   ga += c_dist x gz - p x gout . values_ij,  gq += gz k_j;   and ga += gout . upool once per atom
// (the coefficient gradient as in the recomputing backward, reference quirk included).  Block = (atom, up to eight heads), lane =
// (head, four of the 16 components), so that a row of keys, values or value encodings is one contiguous 512-byte read: a lane
// that took a whole head's 64 bytes would touch a cache line per lane and load, and the tags of the L1 cache set the pace (12
// LDG.128 x 32 lines for 32 pairs of a head).  The dot products meet over four lanes.  Eight warps share the atom's pairs, one
// pair at a time each: latency is covered by warps (64 registers, 32 warps per SM), which does better than two or four pairs in
// flight per warp.  Bound by the latency of the reads.  Per launch, 256 log-normal crystals 49 -> 27 us (two pairs in flight 38),
// 16 cells of 100-200 atoms 145 -> 72 us (111).
// HB: heads side by side; with fewer than eight the rest of a warp takes other pairs of the atom, WA warps an atom, and a block
// 8 / WA atoms: 16 pairs of an atom in flight.  With the column pass behind it, a warp per (atom, head) and lane = pair / eight
// lanes groups of which those beyond the last head idle / this: one head, 256 log-normal crystals 12.6 / 18.3 / 11.9 us, 1 024
// 33 / 58 / 29, 16 cells of 100-200 atoms 22.5 / 44 / 18.8; two heads, 1 024 crystals 72 / 76 / 54; four 113 / 93 / 91.
constexpr int kBsWarps = 8;

__device__ __forceinline__ float quad_sum(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

__device__ __forceinline__ float dot4(const float4 a, const float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }

template <int HB, int WA>
__global__ void __launch_bounds__(kBsWarps * 32) attn_bwd_saved_kernel(const AtArgs A, const Params P)
{
    wait_for_predecessors();
    constexpr int kAtoms = kBsWarps / WA, kSub = 8 / HB;    // atoms of a block, WA warps each; pairs side by side in a warp
    constexpr int kSlots = WA * kSub;                       // pairs of an atom in flight
    const int H = P.H, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t ia = (int64_t)blockIdx.x * kAtoms + warp / WA;
    const int64_t i = kAtoms == 1 ? ia : min(ia, A.N - 1);                         // warps beyond the last atom repeat it
    const int h = blockIdx.y * HB + (lane >> 2) % HB;
    const bool live = kAtoms == 1 || ia < A.N;
    const int64_t ih = i * H + h;
    const int c0 = (lane & 3) * 4;
    auto load4 = [&](const float* src, const int64_t row) { return __ldg(reinterpret_cast<const float4*>(src + row * kAtHd + c0)); };
    const float4 q = load4(A.qs, ih), g = load4(A.gout, ih);
    const float D = quad_sum(dot4(g, load4(A.out, ih)));
    const float lse = __ldg(A.lse + ih);
    const int64_t e0 = A.e_start[i], e1 = A.e_start[i + 1];
    const int64_t j0 = e1 > e0 ? A.edges[A.E + e0] : 0;
    float4 gq = make_float4(0.f, 0.f, 0.f, 0.f);
    float ga = 0.f;
#pragma unroll 1
    for (int64_t e_w = e0 + warp % WA * kSub; e_w < e1; e_w += kSlots) {
        const bool on = kSub == 1 || e_w + (lane >> 2) / HB < e1;
        const int64_t e = kSub == 1 ? e_w : min(e_w + (lane >> 2) / HB, e1 - 1), j = j0 + (e - e0);
        const float4 k = load4(A.k, j * H + h), v = load4(A.v, j * H + h), x = load4(A.val, e * H + h);
        const float z = __ldg(A.z_in + e * H + h), px = __ldg(A.px + e * H + h);
        const float qk = quad_sum(dot4(q, k)), gov = quad_sum(dot4(g, v)), cB = quad_sum(dot4(g, x));
        const float p = __expf(qk + z - lse);
        const float gz = p * (gov + cB - D);
        if (on) {
            if (live && (lane & 3) == 0) A.gz[e * H + h] = gz;
            ga += px * fmaf(P.c_dist, gz, -p * cB);
            gq.x = fmaf(gz, k.x, gq.x); gq.y = fmaf(gz, k.y, gq.y); gq.z = fmaf(gz, k.z, gq.z); gq.w = fmaf(gz, k.w, gq.w);
        }
    }
    // an atom's parts, by its pairs modulo the slots, in a fixed order; the first warp takes all atoms and heads of the block
    __shared__ float part[kBsWarps][5][32];
    part[warp][0][lane] = gq.x; part[warp][1][lane] = gq.y; part[warp][2][lane] = gq.z; part[warp][3][lane] = gq.w;
    part[warp][4][lane] = ga;
    __syncthreads();
    if (warp > 0) return;
    const int atom = lane / (4 * HB);                       // (its head is this lane's own)
    const int64_t io = kAtoms == 1 ? i : (int64_t)blockIdx.x * kAtoms + atom;
    if (atom >= kAtoms || io >= A.N) return;
    auto at = [&](const int c, const int s) { return part[atom * WA + s / kSub][c][s % kSub * 4 * HB + lane % (4 * HB)]; };
    float r[5];
#pragma unroll
    for (int c = 0; c < 5; c++) {
        static_assert(kSlots == 8 || kSlots == 16, "");
        r[c] = ((at(c, 0) + at(c, 1)) + (at(c, 2) + at(c, 3))) + ((at(c, 4) + at(c, 5)) + (at(c, 6) + at(c, 7)));
        if (kSlots == 16)
            r[c] += ((at(c, 8) + at(c, 9)) + (at(c, 10) + at(c, 11))) + ((at(c, 12) + at(c, 13)) + (at(c, 14) + at(c, 15)));
    }
    const int64_t oh = io * H + h;
    const float4 go = kAtoms == 1 ? g : load4(A.gout, oh), up = load4(A.upool, oh);
    const unsigned quad = 0xfu << (lane & ~3);
    float gup = dot4(go, up);
    gup += __shfl_xor_sync(quad, gup, 1);
    gup += __shfl_xor_sync(quad, gup, 2);
    *reinterpret_cast<float4*>(A.gq + oh * kAtHd + c0) = make_float4(r[0], r[1], r[2], r[3]);
    if ((lane & 3) == 0) A.ga[oh] = r[4] + gup;
}

template <int HB, int WA>
static void launch_bwd_saved(const AtArgs& A, const Params& P, cudaStream_t st)
{
    constexpr int atoms = kBsWarps / WA;
    launch_ahead(attn_bwd_saved_kernel<HB, WA>, dim3((unsigned)((A.N + atoms - 1) / atoms), (unsigned)(P.H / HB)), kBsWarps * 32, 0, st,
                 A, P);
}

// blocks per head: the resident ones of the device, no more than the head's atoms can feed
static int at_grid_x(int64_t N, int H, int mode)
{
    const int warps = fw_warps(mode);
    int64_t want = ((int64_t)sm_count() * fw_blocks(mode)) / H;
    if (want < 1) want = 1;
    const int64_t need = (N + warps - 1) / warps;
    if (need < want) want = need < 1 ? 1 : need;
    return (int)want;
}

// blocks per head of the kernels that take pairs one after the other, and of attn_ordered_kernel
static int pairwise_grid_x(int64_t N, int H)
{
    int64_t want = (int64_t)sm_count() * 2 / H;
    if (want < 1) want = 1;
    const int64_t need = (N + 7) / 8;
    if (need < want) want = need < 1 ? 1 : need;
    return (int)want;
}

// Workers per head that the queue of a weighted-PCA training batch is cut for.  An atom's chunks are summed apart, so where the
// cuts are is part of the result: this goes by the device and the batch alone, whatever shape the forward is launched in (it
// was the number of warps of the first kernel that walked such a queue).
static int ordered_plan_workers(int64_t N, int H)
{
    int64_t blocks = (int64_t)sm_count() * 2 / H;
    if (blocks > (N + 7) / 8) blocks = (N + 7) / 8;
    return (int)(blocks < 1 ? 1 : blocks) * 12;
}

// thread = (queue entry, head): the task table.  Entry (x, y, z, w) = atom, result row (the atom, or N + partial row of
// a chunk), offset of the first pair within the atom's pairs, pairs | chunks in use << 24 | (chunk == 1) << 28;
// w = 0: nothing to do.  split: the chunked queue of atom_order_kernel (chunks 1.. in the first kSplitSlots entries,
// then the atoms).
__global__ void __launch_bounds__(256) attn_plan_kernel(const int32_t* __restrict__ order, const int32_t* __restrict__ split,
                                                        const float* __restrict__ a_ik, const int64_t* __restrict__ e_start,
                                                        int64_t N, int64_t n_entries, int H, float scale, int* __restrict__ chunk_count,
                                                        int4* __restrict__ tasks)
{
    wait_for_predecessors();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y;
    if (t >= n_entries) return;
    int4 d = make_int4(0, 0, 0, 0);
    const int info = __ldg(split + 4 + 2 * t);
    if (info != 0) {
        const int i = __ldg(order + t);
        const int chunks = (info >> 4) & 15, index = info & 15;
        const int pairs = (int)(e_start[i + 1] - e_start[i]);
        int active = 1;
        if (chunks > 1)
            active = split_active_chunks(__ldg(a_ik + (int64_t)i * H + h), pairs, __int_as_float(__ldg(split + 4 + 2 * t + 1)),
                                         __int_as_float(__ldg(split + 1)) * scale, chunks);
        if (index < active && pairs > 0) {
            const int lo = pairs * index / active, hi = pairs * (index + 1) / active;
            d.x = i;
            d.y = active > 1 ? (int)N + (info >> 8) + index : i;
            d.z = lo;
            d.w = (hi - lo) | (active << 24) | ((index == 1 ? 1 : 0) << 28);
        }
    }
    if (t >= kSplitSlots) {
        tasks[(size_t)h * n_entries + t] = d;                    // an atom's entry keeps its place
    } else if (d.w != 0) {
        // chunk entries in use gather at the end of the chunk region, in any order (they are all about one target long)
        const int pos = atomicAdd(chunk_count + h, 1);
        tasks[(size_t)h * n_entries + (kSplitSlots - 1 - pos)] = d;
    }
}

// warp = (entry of the queue's chunk region, head): where the entry is chunk 1 of a task (so the task was cut), the
// chunks' results are combined in chunk order.  Forward: chunk c holds the attention output, pooled basis and
// log-sum-exp over its own pairs; the whole is their average weighted by exp(lse_c - lse).
__global__ void __launch_bounds__(256) attn_merge_fwd_kernel(const AtArgs A, const int H)
{
    wait_for_predecessors();
    const int lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int h = blockIdx.y;
    if (t >= kSplitSlots || t < kSplitSlots - __ldg(A.chunk_count + h)) return;
    const int4 d = __ldg(A.tasks + (size_t)h * A.n_entries + t);
    const int active = (d.w >> 24) & 15;
    if (!((d.w >> 28) & 1)) return;
    const int64_t i = d.x, r0 = d.y - A.N - 1;
    float m = -INFINITY;
    for (int c = 0; c < active; c++) m = fmaxf(m, __ldg(A.part_lse + (r0 + c) * H + h));
    float wsum = 0.f;
    for (int c = 0; c < active; c++) wsum += __expf(__ldg(A.part_lse + (r0 + c) * H + h) - m);
    float o = 0.f, s[8];
#pragma unroll
    for (int r = 0; r < 8; r++) s[r] = 0.f;
    for (int c = 0; c < active; c++) {
        const float w = __expf(__ldg(A.part_lse + (r0 + c) * H + h) - m) / wsum;
        if (lane < kAtHd) o = fmaf(w, __ldg(A.part_out + ((r0 + c) * H + h) * kAtHd + lane), o);
        const float* sp = A.part_spool + ((r0 + c) * H + h) * kAtK;
#pragma unroll
        for (int r = 0; r < 8; r++) s[r] = fmaf(w, __ldg(sp + r * 32 + lane), s[r]);
    }
    if (lane == 0) A.lse[i * H + h] = m + logf(wsum);
    if (lane < kAtHd) A.out[(i * H + h) * kAtHd + lane] = o;
    if (A.upool != nullptr && lane < kAtHd) {
        float u = 0.f;
        for (int c = 0; c < active; c++)
            u = fmaf(__expf(__ldg(A.part_lse + (r0 + c) * H + h) - m) / wsum, __ldg(A.part_upool + ((r0 + c) * H + h) * kAtHd + lane), u);
        A.upool[(i * H + h) * kAtHd + lane] = u;
    }
#pragma unroll
    for (int r = 0; r < 8; r++) A.spool[(i * H + h) * kAtK + r * 32 + lane] = s[r];
}

// Backward: the chunks' parts of the query gradient and of the coefficient gradient are summed in chunk order.
__global__ void __launch_bounds__(256) attn_merge_bwd_kernel(const AtArgs A, const int H)
{
    wait_for_predecessors();
    const int lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int h = blockIdx.y;
    if (t >= kSplitSlots || t < kSplitSlots - __ldg(A.chunk_count + h)) return;
    const int4 d = __ldg(A.tasks + (size_t)h * A.n_entries + t);
    const int active = (d.w >> 24) & 15;
    if (!((d.w >> 28) & 1)) return;
    const int64_t i = d.x, r0 = d.y - A.N - 1;
    float gq = 0.f, ga = 0.f;
    for (int c = 0; c < active; c++) {
        if (lane < kAtHd) gq += __ldg(A.part_gq + ((r0 + c) * H + h) * kAtHd + lane);
        ga += __ldg(A.part_ga + (r0 + c) * H + h);
    }
    if (lane == 0) A.ga[i * H + h] = ga;
    if (lane < kAtHd) A.gq[(i * H + h) * kAtHd + lane] = gq;
}

// the task table of one layer (both directions use it); scale: chunks are that many times the queue's target long.
// chunk_count: zeros on entry
int attn_plan(const int32_t* order, const int32_t* split, const float* a_ik, const int64_t* e_start, int64_t N,
              int64_t n_entries, int H, float scale, int* chunk_count, int4* tasks, cudaStream_t st)
{
    if (n_entries <= 0) return CFB200_OK;
    launch_ahead(attn_plan_kernel, dim3((unsigned)((n_entries + 255) / 256), H), 256, 0, st,
                 order, split, a_ik, e_start, N, n_entries, H, scale, chunk_count, tasks);
    return cudaGetLastError() == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

template <int AH, bool TASKS, int MODE, bool EACH = false>
static int launch_tile(const AtArgs& A, const Params& P, cudaStream_t st)
{
    auto kern = attn_tile_kernel<AH, TASKS, MODE, EACH>;
    constexpr size_t smem = fw_smem_bytes(AH, MODE, EACH);
    static std::atomic<bool> attr_done[64];   // per instantiation and device
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return CFB200_E_CUDA;
        attr_done[dev & 63] = true;
    }
    launch_ahead(kern, dim3(at_grid_x(TASKS ? A.N * kSplitMaxChunks : A.N, P.H, MODE), P.H), fw_warps(MODE) * 32, smem, st,
                 A, P);
    if (TASKS) {
        const dim3 grid(kSplitSlots / 8, P.H);
        if (MODE == 2) launch_ahead(attn_merge_bwd_kernel, grid, 256, 0, st, A, P.H);
        else launch_ahead(attn_merge_fwd_kernel, grid, 256, 0, st, A, P.H);
    }
    return cudaGetLastError() == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

template <bool ANG, bool TASKS>
static int launch_pairwise(const AtArgs& A, const Params& P, cudaStream_t st)
{
    auto kern = attn_pairwise_kernel<ANG, TASKS>;
    static std::atomic<bool> attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPwSmem) != cudaSuccess) return CFB200_E_CUDA;
        attr_done[dev & 63] = true;
    }
    launch_ahead(kern, dim3(pairwise_grid_x(A.N, P.H), P.H), kPwWarps * 32, kPwSmem, st, A, P);
    if (TASKS) launch_ahead(attn_merge_fwd_kernel, dim3(kSplitSlots / 8, P.H), 256, 0, st, A, P.H);
    return cudaGetLastError() == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

template <bool TASKS>
static int launch_ordered(const AtArgs& A0, const Params& P, cudaStream_t st)
{
    AtArgs A = A0;
    A.vec = on_grid({A.qs, A.k});
    auto kern = attn_ordered_kernel<TASKS>;
    static std::atomic<bool> attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOrSmem) != cudaSuccess) return CFB200_E_CUDA;
        attr_done[dev & 63] = true;
    }
    launch_ahead(kern, dim3(pairwise_grid_x(A.N, P.H), P.H), kOrWarps * 32, kOrSmem, st, A, P);
    if (TASKS) launch_ahead(attn_merge_fwd_kernel, dim3(kSplitSlots / 8, P.H), 256, 0, st, A, P.H);
    return cudaGetLastError() == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

template <int MODE>
static int launch_tile(const AtArgs& A0, const Params& P, cudaStream_t st)
{
    AtArgs A = A0;
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    A.vec = aligned(A.qs) && aligned(A.k) && aligned(A.val) && aligned(A.gout) && aligned(A.v);
    A.vec_list = aligned(A.list);
    if (!A.counters_zeroed && cudaMemsetAsync(A.counters, 0, sizeof(int) * P.H, st) != cudaSuccess) return CFB200_E_CUDA;
    const bool tasks = A.tasks != nullptr;
    if (A.W[1] == nullptr) {
        // the plain backward: sums of eight pairs at once pay in big cells (more than 32 pairs per atom), with the task table
        if (MODE == 2 && tasks && A.E <= 32 * A.N) return launch_tile<0, true, MODE, MODE == 2>(A, P, st);
        return tasks ? launch_tile<0, true, MODE>(A, P, st) : launch_tile<0, false, MODE, MODE == 2>(A, P, st);
    }
    if (P.angle_dim <= 32) return tasks ? launch_tile<1, true, MODE>(A, P, st) : launch_tile<1, false, MODE>(A, P, st);
    return tasks ? launch_tile<2, true, MODE>(A, P, st) : launch_tile<2, false, MODE>(A, P, st);
}

// A.val set: the forward leaves per-pair results for attn_fused_bwd.
int attn_fused_fwd(const AtArgs& A, const Params& P, cudaStream_t st)
{
    if (A.N == 0) return CFB200_OK;
    // Without lists the training forward sweeps each pair's box for the smallest distance, then for weights and records; in
    // tiles the normaliser takes a third sweep and the records a detour (a training step of 256 log-normal crystals without
    // lists 5.5 against 6.3 ms).
    if (A.val != nullptr && (A.pairwise || A.list == nullptr)) {
        if (!A.counters_zeroed && cudaMemsetAsync(A.counters, 0, sizeof(int) * P.H, st) != cudaSuccess) return CFB200_E_CUDA;
        if (A.list != nullptr && A.W[1] != nullptr) return A.tasks != nullptr ? launch_ordered<true>(A, P, st) : launch_ordered<false>(A, P, st);
        if (A.tasks != nullptr) return A.W[1] != nullptr ? launch_pairwise<true, true>(A, P, st) : launch_pairwise<false, true>(A, P, st);
        return A.W[1] != nullptr ? launch_pairwise<true, false>(A, P, st) : launch_pairwise<false, false>(A, P, st);
    }
    return A.val != nullptr ? launch_tile<1>(A, P, st) : launch_tile<0>(A, P, st);
}

// A.val set: from the per-pair results of the forward; else by recomputing the lattice sums.
int attn_fused_bwd(const AtArgs& A, const Params& P, cudaStream_t st)
{
    if (A.N == 0) return CFB200_OK;
    if (A.val == nullptr) return launch_tile<2>(A, P, st);
    if (!on_grid({A.qs, A.k, A.v, A.gout, A.out, A.upool, A.val, A.gq})) return CFB200_E_SHAPE;
    if (P.H % 8 == 0) launch_bwd_saved<8, 8>(A, P, st);             // (the heads are a power of two)
    else if (P.H == 4) launch_bwd_saved<4, 8>(A, P, st);
    else if (P.H == 2) launch_bwd_saved<2, 4>(A, P, st);
    else launch_bwd_saved<1, 2>(A, P, st);
    return cudaGetLastError() == cudaSuccess ? CFB200_OK : CFB200_E_CUDA;
}

}  // namespace cfb
