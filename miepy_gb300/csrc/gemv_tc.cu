// Tensor-core (tcgen05) matrix pass of the packed operator, for blocks of R = 4 or
// 8 right-hand sides (polarisations x sources) of the FP32 inner solves.
//
// Replaces, for multi-RHS blocks, the row-block GEMV of the reference's
// solve_linear_system (cpp/src/interactions.cpp:70-92, ParallelDenseMatrix::
// scaleAndAddTo): with R right-hand sides a pass streams each matrix block once and
// multiplies it by 2R vectors (the block serves both block rows, see solve.cu), so
// the CUDA-core FP32 pipe runs out before HBM does; the tensor cores do not.
//
// Arithmetic: split-BF16x3.  Each complex64 matrix element a is held as two bf16
// planes, hi = bf16(a) and lo = bf16(a - hi) per real component (k_tc_tiles, once
// per assembly), and each vector element z likewise; the product is
// A_hi z_hi + A_hi z_lo + A_lo z_hi, accumulated in FP32 in tensor memory: about
// 5e-6 relative to the largest term, against 4e-7 for complex64 arithmetic.  The
// mixed method's FP32 inner solves (to 1e-4) use it; its refinement residuals keep
// the CUDA-core complex64 and double-float passes.
//
// Half of a block is read: with P, Q its upper quadrants (block = [[P, Q], [Q, P]] over
// the polarisations) the tiles hold P + Q and P - Q, which act on (z1 +- z2) / 2, z1 and z2
// the two polarisations of a vector z.  A complex product as a real GEMM: a tile is
// [B/2 rows][B real columns] (re, im interleaved along K); a complex vector becomes two
// real B-operand rows, (re z, -im z) giving re(A z) and (im z, re z) giving im(A z).  For
// both signs one MMA per K-step multiplies A_hi by N = 16R rows [U_h+ W_h+ U_h- W_h- | U_l+
// W_l+ U_l- W_l-] and a second A_lo by the first 8R, into an accumulator of N FP32 columns;
// of the tile's planes (+ hi, + lo, - hi, - lo, their rows one after the other) the first
// MMA's 128 rows hold + hi and, from row 2 Hp on, - hi, the second's + lo and - lo at the
// same rows, and only the columns of a row's own sign are read out:
//   U = A z_j (row product of block (i, j)),
//   W = A w_i (column product), w_i = S z_i,
// with z[s] = eps(s) y[rho(s)] of the solver's y vectors.  k_yprep_tc writes each particle's
// rows of U and of W once per product as bf16 pieces in the operand's layout, so that a
// block's operand arrives by copies.  The results C[rho(r)] = eps(r) (A z)[r] are stored
// by sign as the CUDA-core pass stores its +- column sums: C[s] = c+ + c-, C[rmax + s] =
// c+ - c- with c+ = eps (the sum of sign -) and c- = eps (that of sign +), as eps of the
// two polarisations are opposite; element (column, right-hand side q) of a term lies at 16-byte
// word (q / 2) B + sign rmax + column, so that a warp's stores are contiguous.
//
// Work unit: a rectangle of up to 4 rows x several columns of blocks, column by column, its
// row sums (of all its columns) and the column's sums kept in registers: the partials of a
// block by itself are a third of its tile's bytes at R = 8, B = 48, and went through HBM both
// in this pass and in the reduce (N = 200, lmax 4, R = 8: 92 MB a product; with rectangles
// 25 MB, the product 56 us against 79).
//
// Pipeline per CTA (6 warps, two CTAs per SM where their stages fit, persistent over
// units), each role running ahead of the next one as far as the rings let it: a producer
// warp copies, per block, the tile and the operand's pieces (TMA bulk copies) into a ring
// of stages, with a job record; one thread issues the block's MMAs (M = 128: the rows past
// the tile's read what follows it and are discarded) into one of two accumulators; the
// warps of the tile's rows read the accumulator (tcgen05.ld) and add it to the sums.  Every wait is bounded; an expired wait sets the error flag and the
// abort flag, which ends the other roles' waits, and the CTA waits (again bounded) for its
// copies and MMAs in flight before it frees its TMEM and exits.
//
// Bound: per block, the issue of 9 copies (270 cycles) and of the MMAs and the copies' bytes
// from L2 (the operand's 12 KB with the tile's 9 KB at R = 8, B = 48), next to the tiles' 27
// us at the measured copy rate.  N = 200, lmax 4: 42 us at R = 8, 35 at R = 4; with whole
// blocks, their operand built by each CTA, 102 and 89.  (Issued from divergent code, copies
// and MMAs took 83 to 160 cycles each: 71 and 57 us; a sign at a time, with twice the MMAs,
// each bound by its 128 rows: 49 and 36.)
#include <cuda_bf16.h>

#include "gb_common.cuh"
#include "gb_internal.h"
#include "solve_plan.cuh"

namespace {

constexpr int kTcThreads = 192;   // warps 0-3: accumulator rows out; 4: copies in; 5: MMAs
constexpr int kTcMaxStages = 5;
constexpr long long kTcWaitCycles = 400000000LL;   // about 0.2 s of SM clock

__device__ __forceinline__ unsigned su32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void pdl_wait_tc() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger_tc() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// ----------------------------------------------------------------- mbarrier --
__device__ __forceinline__ void bar_init(uint64_t* b, unsigned n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded; given a flag, it also ends (false) once the flag is set
__device__ __forceinline__ bool bar_wait(uint64_t* b, unsigned parity, const volatile int* stop = nullptr) {
    if (bar_try(b, parity)) return true;
    const long long t0 = clock64();
    while (!bar_try(b, parity))
        if ((stop && *stop) || clock64() - t0 > kTcWaitCycles) return false;
    return true;
}
// one lane of the warp (the same one each time); warp-uniform code around it keeps the
// operands of the copies and MMAs in uniform registers
__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes, uint64_t* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     su32(dst)),
                 "l"(src), "r"(bytes), "r"(su32(b))
                 : "memory");
}
__device__ __forceinline__ void bulk_copy_hint(void* dst, const void* src, unsigned bytes, uint64_t* b, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::"r"(
            su32(dst)),
        "l"(src), "r"(bytes), "r"(su32(b)), "l"(pol)
        : "memory");
}
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol));
    return pol;
}

// ------------------------------------------------------------------ tcgen05 --
__device__ __forceinline__ void tmem_alloc(unsigned* slot, unsigned ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(su32(slot)), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, bf16 inputs, FP32 accumulation (kind::f16)
__device__ __forceinline__ void mma_bf16(unsigned d, uint64_t a, uint64_t b, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on the mbarrier once every MMA this thread issued before has completed
__device__ __forceinline__ void mma_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(su32(b))
                 : "memory");
}
// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows x
// 16 bytes; lbo = byte step between core matrices along K, sbo = along M (or N).
__device__ __forceinline__ uint64_t smem_desc(unsigned saddr, unsigned lbo, unsigned sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}
// Instruction descriptor of kind::f16: FP32 accumulator, bf16 A and B, both K-major.
__host__ __device__ constexpr unsigned idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(N >> 3) << 17) | ((unsigned)(M >> 4) << 24);
}

// ------------------------------------------------------------ shared layout --
// Header: the barriers, the TMEM address, the abort flag, the consumed count, the job
// records of the stages and of the two accumulators; then the stages, each a block's tile
// (hi, lo of P + Q, then of P - Q) and the operand's pieces (8, 2R rows each).
struct TcJob {
    long long cw;    // first element of the column's partial in CW; -1: no more blocks for this CTA
    long long cu;    // of the unit's first row's partial in CU
    int row;         // the block's row of the unit
    int rows;        // the unit's rows, at its last block, else 0
    int stride;      // elements between the rows' partials
    int last;        // the column's last block
};
// Block k's record lies in slot k % kTcJobs.  It is read by the MMA thread and by the warps
// that read the accumulator out, which are at most kTcMaxStages + 1 blocks behind.
constexpr int kTcJobs = 8;
static_assert(kTcJobs >= kTcMaxStages + 2, "job records");
struct TcHeader {
    uint64_t full[kTcMaxStages], empty[kTcMaxStages];   // a stage's copies landed; its MMAs done
    uint64_t mdone[2], job[2], free[2];                 // an accumulator's MMAs done, job known, read out
    long long consumed;                                 // jobs the MMA thread has taken
    TcJob jobs[kTcJobs];
    unsigned tmem;
    int abort;
};
struct TcLayout {
    unsigned sbo, plane, tile, piece, stage, total;
};
constexpr unsigned kTcStageOff = 512;
static_assert(sizeof(TcHeader) <= kTcStageOff, "header");
__host__ __device__ inline TcLayout tc_layout(int B, int R, int S) {
    TcLayout L;
    L.sbo = (unsigned)gb::tc_cols(B) * 16u;
    L.plane = (unsigned)(gb::tc_rows(B) / 8) * L.sbo;
    L.tile = 4u * L.plane;
    L.piece = (unsigned)(R / 4) * L.sbo;   // 2R rows
    L.stage = L.tile + 8u * L.piece;
    const unsigned end = kTcStageOff + (unsigned)S * L.stage;
    // an M = 128 MMA reads 16 row groups from the first and second plane on
    const unsigned reach = kTcStageOff + (unsigned)(S - 1) * L.stage + L.plane + 16u * L.sbo;
    L.total = end > reach ? end : reach;
    return L;
}

// ------------------------------------------------------------- tile builder --
// mat64 [pairs][B][B] complex64 (the assembler's hi plane; its upper half is read) ->
// bf16 hi/lo tiles of P + Q and P - Q.  blockIdx.y = cluster; CTAs stride over its pairs;
// one thread per (row, 4 complex columns): a 16-byte store into each plane.  Bound by its
// reads and writes: N = 200, lmax 4 59 us (6.2 TB/s), 119 us with whole blocks.
__global__ void __launch_bounds__(256)
k_tc_tiles(const gb::SysDev* __restrict__ sys, const float2* __restrict__ mat64, unsigned char* __restrict__ out) {
    const gb::SysDev S = sys[blockIdx.y];
    const int B = S.B, H = B / 2, KG = gb::tc_cols(B) / 8;
    const long long plane = gb::tc_plane_bytes(B), blk = gb::tc_block_bytes(B);
    const unsigned sbo = (unsigned)gb::tc_cols(B) * 16u;
    const int items = gb::tc_rows(B) * KG;
    for (long long p = blockIdx.x; p < S.P; p += gridDim.x) {
        const float2* src = mat64 + S.mat_off + p * (long long)B * B;
        unsigned char* dst = out + S.tc_off + p * blk;
        for (int it = threadIdx.x; it < items; it += blockDim.x) {
            const int m8 = it & 7, rest = it >> 3, g = rest % KG, m = (rest / KG) * 8 + m8;
            const float2* row = src + (long long)m * B + 4 * g;
            float2 P[4], Q[4];
            if (m < H && 4 * g + 3 < H && H % 2 == 0) {   // 16-byte aligned: B and H are even
                const float4* pv = reinterpret_cast<const float4*>(row);
                const float4* qv = reinterpret_cast<const float4*>(row + H);
                const float4 a = __ldg(pv), b = __ldg(pv + 1), c = __ldg(qv), d = __ldg(qv + 1);
                P[0] = make_float2(a.x, a.y), P[1] = make_float2(a.z, a.w);
                P[2] = make_float2(b.x, b.y), P[3] = make_float2(b.z, b.w);
                Q[0] = make_float2(c.x, c.y), Q[1] = make_float2(c.z, c.w);
                Q[2] = make_float2(d.x, d.y), Q[3] = make_float2(d.z, d.w);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const bool in = m < H && 4 * g + e < H;
                    P[e] = in ? __ldg(row + e) : make_float2(0.f, 0.f);
                    Q[e] = in ? __ldg(row + H + e) : make_float2(0.f, 0.f);
                }
            }
            unsigned char* at = dst + (size_t)(m >> 3) * sbo + (size_t)g * 128 + (size_t)m8 * 16;
#pragma unroll
            for (int s = 0; s < 2; s++) {
                uint4 h, l;
                unsigned* hp = &h.x;
                unsigned* lp = &l.x;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float ax = s ? P[e].x - Q[e].x : P[e].x + Q[e].x, ay = s ? P[e].y - Q[e].y : P[e].y + Q[e].y;
                    const float hr = gb::bf_round(ax), hi = gb::bf_round(ay);
                    hp[e] = gb::bf2(hr, hi);
                    lp[e] = gb::bf2(ax - hr, ay - hi);
                }
                *reinterpret_cast<uint4*>(at + 2 * s * plane) = h;
                *reinterpret_cast<uint4*>(at + (2 * s + 1) * plane) = l;
            }
        }
    }
}

// ------------------------------------------------------------- matrix pass --
// The warp's 32 TMEM lanes of columns a0 .. a0 + NC - 1 and a1 .. a1 + NC - 1 (NC = 8 or
// 16), waited for in the statement that loads them.
template <int NC> __device__ __forceinline__ void tmem_ld_pair(unsigned a0, unsigned a1, unsigned* r);
template <> __device__ __forceinline__ void tmem_ld_pair<8>(unsigned a0, unsigned a1, unsigned* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(a0), "r"(a1)
        : "memory");
}
template <> __device__ __forceinline__ void tmem_ld_pair<16>(unsigned a0, unsigned a1, unsigned* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(a0), "r"(a1)
        : "memory");
}
template <int NC> __device__ __forceinline__ void tmem_ld2(unsigned a0, unsigned a1, float (&v0)[NC], float (&v1)[NC]) {
    unsigned r[2 * NC];
    tmem_ld_pair<NC>(a0, a1, r);
#pragma unroll
    for (int i = 0; i < NC; i++) {
        v0[i] = __uint_as_float(r[i]);
        v1[i] = __uint_as_float(r[NC + i]);
    }
}

// The pass over units [ubeg, uend) of one block size B with S stages.
template <int R>
__global__ void __launch_bounds__(kTcThreads, 2)
k_pgemv_tc(const gb::SysDev* __restrict__ sys, const gb::TcUnit* __restrict__ units, long long ubeg, long long uend, int I,
           const gb::KState* __restrict__ st, int mask, const unsigned char* __restrict__ mat_tc,
           const unsigned char* __restrict__ Yu, const unsigned char* __restrict__ Yw, float2* __restrict__ CU,
           float2* __restrict__ CW, const gb::SysPlan* __restrict__ plan, const long long* __restrict__ tc_rows, int B, int S,
           int* __restrict__ err) {
    constexpr int N = 16 * R;             // columns of an accumulator
    constexpr unsigned NCOL = 2 * N;      // two accumulators (128 or 256: a power of 2 >= 32)
    constexpr unsigned IDESC_FULL = idesc_bf16(128, N);
    constexpr unsigned IDESC_HALF = idesc_bf16(128, N / 2);
    const TcLayout L = tc_layout(B, R, S);
    const int H = B / 2, minus = 2 * gb::tc_rows(B);   // TMEM lane (MMA row) of sign -'s first row
    extern __shared__ __align__(1024) unsigned char sm[];
    TcHeader& hd = *reinterpret_cast<TcHeader*>(sm);
    unsigned char* stages = sm + kTcStageOff;
    volatile int* stop = &hd.abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

    if (tid == 0) {
        for (int q = 0; q < S; q++) {
            bar_init(hd.full + q, 1);
            bar_init(hd.empty + q, 1);
        }
        for (int x = 0; x < 2; x++) {
            bar_init(hd.mdone + x, 1);
            bar_init(hd.job + x, 1);
            bar_init(hd.free + x, (H + 31) / 32 + (minus + H + 31) / 32 - minus / 32);   // the warps that hold rows
        }
        hd.abort = 0;
        hd.consumed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(&hd.tmem, NCOL);
        tmem_relinquish();
    }
    proxy_fence();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const unsigned tmem = hd.tmem;
    pdl_wait_tc();   // operands and solver state come from the preceding kernels
    pdl_trigger_tc();
    auto give_up = [&]() {
        *stop = 1;
        atomicExch(err, 1);
    };

    long long k = 0;   // producer: jobs written
    if (warp == 4) {
        // ------------------------------------------------------------ producer
        // Walks this CTA's units (every gridDim.x-th, skipping clusters with no active
        // right-hand side), the records of 32 of them loaded at once.
        const long long G = gridDim.x;
        const uint64_t pol = evict_first_policy();
        const unsigned pbytes = 4u * L.piece;   // of a particle's operand
        const int BR = B * R;
        gb::TcUnit mine{};
        int at = 32;   // unit of the 32 loaded
        int cur = -1, NP = 0, s = 0;
        unsigned phase = 1;   // of the stage's empty barrier: passes at once the first time round
        bool act = false;
        long long t_off = 0, y_off = 0, cw0 = 0, cu0 = 0, rows0 = 0;
        bool run = true;
        for (long long pw = ubeg + blockIdx.x; run && pw < uend; pw += G) {
            if (at == 32) {
                at = 0;
                if (pw + lane * G < uend) mine = units[pw + lane * G];
            }
            const int sysi = __shfl_sync(0xffffffffu, mine.sys, at), i0 = __shfl_sync(0xffffffffu, mine.i0, at),
                      j0 = __shfl_sync(0xffffffffu, mine.j0, at), nj = __shfl_sync(0xffffffffu, mine.nj, at),
                      c = __shfl_sync(0xffffffffu, mine.c, at), C = __shfl_sync(0xffffffffu, mine.C, at);
            at++;
            if (sysi != cur) {
                cur = sysi;
                act = gb::any_active<R>(st, cur, mask);
                const gb::SysDev& Sd = sys[cur];
                const gb::SysPlan& pl = plan[cur];
                NP = Sd.N;
                t_off = Sd.tc_off;
                y_off = Sd.ty_off * R;
                cw0 = pl.tc_cw;
                cu0 = pl.tc_cu;
                rows0 = pl.tc_base;
            }
            if (!act) continue;
            const int rows = min(I, NP - i0), stride = C * BR;
            const long long cu = cu0 + (tc_rows[rows0 + i0] + c) * BR;
            long long term = tc_rows[rows0 + NP + 1 + j0] + i0 / I;   // the column's partial of this row group
            const unsigned char* usrc = Yu + y_off + (long long)j0 * pbytes;
            const unsigned char* wsrc = Yw + y_off + (long long)i0 * pbytes;
            const unsigned char* tsrc = mat_tc + t_off + (pair_start(i0, NP) + j0 - i0 - 1) * (long long)L.tile;
            for (int jj = 0; run && jj < nj; jj++) {
                const int n = min(rows, j0 + jj - i0);   // the column's blocks
                const long long cw = cw0 + term * BR;
                const unsigned char* ts = tsrc;
                const unsigned char* ws = wsrc;
                for (int ii = 0; ii < n; ii++, k++) {
                    run = __all_sync(0xffffffffu, bar_wait(hd.empty + s, phase, stop));
                    if (!run) break;
                    if (elect_one()) {
                        TcJob J;
                        J.cw = cw;
                        J.cu = cu;
                        J.row = ii;
                        J.rows = ii == n - 1 && jj == nj - 1 ? rows : 0;
                        J.stride = stride;
                        J.last = ii == n - 1;
                        hd.jobs[k % kTcJobs] = J;
                        bar_expect_tx(hd.full + s, L.stage);   // arrive (release): the job record goes with it
                        unsigned char* dst = stages + (size_t)s * L.stage;
                        bulk_copy_hint(dst, ts, L.tile, hd.full + s, pol);
#pragma unroll
                        for (int q = 0; q < 8; q++)   // (hi / lo, sign, U / W)
                            bulk_copy(dst + L.tile + q * L.piece, ((q & 1) ? ws : usrc) + (q >> 1) * L.piece, L.piece,
                                      hd.full + s);
                    }
                    __syncwarp();
                    ts += (long long)(NP - 2 - i0 - ii) * L.tile;   // (i + 1, j)
                    ws += pbytes;
                    if (++s == S) {
                        s = 0;
                        phase ^= 1u;
                    }
                }
                tsrc += L.tile;
                usrc += pbytes;
                term += (j0 + jj + I - 1) / I;   // column j has one per row group that starts above it
            }
        }
        if (!run && lane == 0) give_up();
        if (run && lane == 0) {   // the end: an invalid job, with a plain arrive
            if (bar_wait(hd.empty + s, phase, stop)) {
                hd.jobs[k % kTcJobs].cw = -1;
                bar_arrive(hd.full + s);
                k++;
            } else {
                give_up();
            }
        }
    } else if (warp == 5) {
        // --------------------------------------------------------- MMA issuer
        const int KS = gb::tc_cols(B) / 16;   // <= 5
        long long g = 0;                      // blocks whose MMAs were issued
        int s = 0;
        unsigned phase = 0;
        bool ok = true;
        while (true) {
            const int x = (int)(g & 1);
            // the accumulator read out (block g - 2), the stage's copies landed
            ok = bar_wait(hd.free + x, (unsigned)((g >> 1) & 1) ^ 1u, stop) && bar_wait(hd.full + s, phase, stop);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const bool valid = __all_sync(0xffffffffu, hd.jobs[g % kTcJobs].cw >= 0);
            if (elect_one()) bar_arrive(hd.job + x);
            __syncwarp();
            if (!valid) break;
            tc_after_sync();
            const unsigned a = su32(stages) + (unsigned)s * L.stage, b = a + L.tile;
            const unsigned d = tmem + (unsigned)(x * N);
            const uint64_t da = smem_desc(a, 128, L.sbo), db = smem_desc(b, 128, L.sbo);   // + 16 per 256 bytes
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 5; ks++) {
                    if (ks < KS) {
                        mma_bf16(d, da + 16u * ks, db + 16u * ks, IDESC_FULL, ks > 0);
                        mma_bf16(d, da + 16u * ks + (L.plane >> 4), db + 16u * ks, IDESC_HALF, 1);
                    }
                }
                mma_commit(hd.mdone + x);
                mma_commit(hd.empty + s);   // the stage is free once these MMAs have read it
            }
            __syncwarp();
            g++;
            if (++s == S) {
                s = 0;
                phase ^= 1u;
            }
        }
        if (lane == 0) hd.consumed = ok ? g + 1 : g;
        if (!ok && lane == 0) {
            give_up();
            for (long long e = (g >= 2 ? g - 2 : 0); e < g; e++)   // bounded waits for the MMAs still in flight
                (void)bar_wait(hd.mdone + (e & 1), (unsigned)((e >> 1) & 1));
        }
    } else if (warp * 32 < H || (warp * 32 + 31 >= minus && warp * 32 < minus + H)) {
        // ---------------------------------------------------- accumulators out
        const int sig = warp * 32 < H ? 0 : 1, m = tid - sig * minus;   // sign (of all the warp's rows), row
        const bool row = m >= 0 && m < H;
        int at = 0;          // its 16-byte word in a term: column rho(m) of the other sign
        unsigned eneg = 0;
        if (row) {
            const int info = __ldg(sys[units[ubeg].sys].rowinfo + m);   // every cluster of the launch has block size B
            at = (sig ^ 1) * H + (info & ((1 << 29) - 1));
            eneg = (info >> 29) & 1;
        }
        const unsigned taddr = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(sig * 4 * R);
        float u[gb::kTcRows][2 * R], w[2 * R];   // sums of the unit's rows, of the column
#pragma unroll
        for (int q = 0; q < 2 * R; q++) {
            w[q] = 0.f;
#pragma unroll
            for (int t = 0; t < gb::kTcRows; t++) u[t][q] = 0.f;
        }
        auto put = [&](float2* to, float (&v)[2 * R]) {   // a partial out, its sums back to zero
            float4* p = reinterpret_cast<float4*>(to) + at;
#pragma unroll
            for (int q = 0; q < 2 * R; q += 4) {
                if (row)
                    p[q / 4 * B] = make_float4(flipf(v[q], eneg), flipf(v[q + 1], eneg), flipf(v[q + 2], eneg),
                                               flipf(v[q + 3], eneg));
                v[q] = v[q + 1] = v[q + 2] = v[q + 3] = 0.f;
            }
        };
        for (long long e = 0;; e++) {
            const int x = (int)(e & 1);
            const unsigned phase = (unsigned)((e >> 1) & 1);
            bool ok = bar_wait(hd.job + x, phase, stop);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (lane == 0) give_up();
                break;
            }
            const TcJob J = hd.jobs[e % kTcJobs];
            if (J.cw < 0) break;   // the same record for every lane
            ok = bar_wait(hd.mdone + x, phase, stop);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (lane == 0) give_up();
                break;
            }
            tc_after_sync();
            float h[2 * R], l[2 * R];   // of z_h and of z_l
            const unsigned ta = taddr + (unsigned)(x * N);
            tmem_ld2<2 * R>(ta, ta + 8 * R, h, l);
#pragma unroll
            for (int t = 0; t < gb::kTcRows; t++)
                if (J.row == t) {
#pragma unroll
                    for (int q = 0; q < 2 * R; q++) u[t][q] += h[q] + l[q];
                }
            tmem_ld2<2 * R>(ta + 2 * R, ta + 10 * R, h, l);
            tc_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(hd.free + x);
#pragma unroll
            for (int q = 0; q < 2 * R; q++) w[q] += h[q] + l[q];
            if (J.last) put(CW + J.cw, w);
            if (J.rows) {
#pragma unroll
                for (int t = 0; t < gb::kTcRows; t++)
                    if (t < J.rows) put(CU + J.cu + (long long)t * J.stride, u[t]);
            }
        }
    }
    tc_before_sync();
    __syncthreads();
    if (warp == 4 && lane == 0)   // drain: copies of jobs written and not taken (bounded waits)
        for (long long q = hd.consumed; q < k; q++) (void)bar_wait(hd.full + (q % S), (unsigned)((q / S) & 1));
    __syncthreads();
    if (warp == 0) {
        tc_after_sync();
        tmem_dealloc(tmem, NCOL);
    }
}

}   // namespace

namespace gb {

int launch_pgemv_tc(int R, const SysDev* sys, const TcUnit* units, long long ubeg, long long uend, int I,
                    const KState* st, int mask, const void* mat_tc, const void* Yu, const void* Yw, void* CU, void* CW,
                    const SysPlan* plan, const long long* tc_rows, int B, int* err, cudaStream_t stream) {
    if (uend <= ubeg) return GB_OK;
    if (R != 4 && R != 8) return gb_set_error(GB_UNSUPPORTED, "tensor-core pass: R must be 4 or 8 (got %d)", R);
    if (B > 70) return gb_set_error(GB_UNSUPPORTED, "tensor-core pass: block size %d > 70 (lmax 5)", B);
    if ((reinterpret_cast<uintptr_t>(mat_tc) | reinterpret_cast<uintptr_t>(Yu) | reinterpret_cast<uintptr_t>(Yw)) & 15)
        return gb_set_error(GB_BAD_ARG, "tensor-core pass: matrix and y vectors must be 16-byte aligned");
    // as many stages as let two CTAs share an SM (228 KB, 1 KB of them reserved per CTA): 3 at
    // B = 70, 5 up to B = 48
    int S = kTcMaxStages;
    while (S > 3 && 2u * (tc_layout(B, R, S).total + 1024u) > 228u * 1024u) S--;
    const TcLayout L = tc_layout(B, R, S);
    const void* kfn = R == 4 ? reinterpret_cast<const void*>(k_pgemv_tc<4>) : reinterpret_cast<const void*>(k_pgemv_tc<8>);
    GB_CUDA_TRY(ensure_dynamic_smem(kfn, L.total));
    const long long n = uend - ubeg;
    const long long grid = n < 2LL * sm_count() ? n : 2LL * sm_count();
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = L.total;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    note_launch();
    const unsigned char* m = static_cast<const unsigned char*>(mat_tc);
    const unsigned char* yu = static_cast<const unsigned char*>(Yu);
    const unsigned char* yw = static_cast<const unsigned char*>(Yw);
    float2* cu = static_cast<float2*>(CU);
    float2* cw = static_cast<float2*>(CW);
    if (R == 4)
        GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_pgemv_tc<4>, sys, units, ubeg, uend, I, st, mask, m, yu, yw, cu, cw, plan,
                                       tc_rows, B, S, err));
    else
        GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_pgemv_tc<8>, sys, units, ubeg, uend, I, st, mask, m, yu, yw, cu, cw, plan,
                                       tc_rows, B, S, err));
    return GB_OK;
}

}   // namespace gb

extern "C" {

size_t gb_tc_matrix_bytes(int nsys, const gb_system* sys) {
    if (nsys < 1 || !sys) return 0;
    std::vector<gb::SysDev> sd;
    if (gb::make_sysdev(nsys, sys, 0, sd)) return 0;
    const gb::SysDev& last = sd.back();
    return (size_t)(last.tc_off + last.P * gb::tc_block_bytes(last.B));
}

int gb_tc_matrix_build(int nsys, const gb_system* sys, const float* mat64, void* mat_tc, void* stream) {
    if (nsys < 1 || !sys || !mat64 || !mat_tc) return gb_set_error(GB_BAD_ARG, "null argument");
    if (reinterpret_cast<uintptr_t>(mat64) & 15 || reinterpret_cast<uintptr_t>(mat_tc) & 15)
        return gb_set_error(GB_BAD_ARG, "matrices must be 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<gb::SysDev> sd;
    int e = gb::make_sysdev(nsys, sys, s, sd);
    if (e) return e;
    if (nsys > 65535) return gb_set_error(GB_UNSUPPORTED, "more than 65535 clusters in one batch");
    long long maxP = 0;
    for (const gb::SysDev& d : sd) maxP = d.P > maxP ? d.P : maxP;
    if (maxP == 0) return GB_OK;
    void* dsys = nullptr;
    int slot = 0;
    e = gb::stage_acquire(sd.data(), sizeof(gb::SysDev) * sd.size(), s, &dsys, &slot);
    if (e) return e;
    const unsigned gx = (unsigned)(maxP < 4096 ? maxP : 4096);
    gb::note_launch();
    k_tc_tiles<<<dim3(gx, (unsigned)nsys), 256, 0, s>>>(static_cast<const gb::SysDev*>(dsys),
                                                         reinterpret_cast<const float2*>(mat64),
                                                         static_cast<unsigned char*>(mat_tc));
    GB_CUDA_TRY(cudaGetLastError());
    return gb::stage_release(slot, s);
}

}   // extern "C"
