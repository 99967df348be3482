// Tensor-core linear kernel for prefill and large batches (M > 16), sm_100a:
//   out[M,N] = x[M,K] . W[N,K]^T, fp16 operands, fp32 accumulation in tensor memory.
//
// Stands in for the reference's M > 1 path, a CLBlast Gemm<cl_half> call
// (src/models/lfm2-5-350m/src/utils.cpp:1334-1345: RowMajor, A no-trans, B trans,
// lda = ldb = K, ldc = N, alpha 1, beta 0), for its token-by-token loop over
// quantised weights (src/models/lfm2-5-350m/src/model.cpp:243-251), and for the element-wise
// kernels that follow those GEMMs in its layers (bias, residual, SiLU-multiply).
//
// A block computes tiles of 128 weight rows x bn tokens (bn <= 256, a multiple of 16), the weights
// as the MMA's M operand, into tensor memory:
//   * warp 0: TMA producer of the token operand (64-wide K blocks, 128-byte swizzle) and,
//     for fp16 weights, of the weight operand.
//   * warp 1: issues tcgen05.mma (cta_group::1, kind::f16, M128 x N(bn) x K16, four per
//     K block and weight); tcgen05.commit hands operands back and signals the epilogue.
//   * warps 2-9 (Q4: 2-5): epilogue.  Warp w reads lanes 32 (w % 4) .. +31 of the accumulator with
//     tcgen05.ld (lane = weight row, column = token) and finishes the values there: int8 row
//     scale, bias, in-place residual, SiLU gate.  SwiGLU: a tile is 64 gate rows and the 64 up rows of
//     the same numbers, and the warps that hold them swap half of each other's columns through shared
//     memory, so that every thread finishes SiLU(gate) * up for one row and half of the tokens.
//   * int8 / Q4 weights are streamed packed, once, in spans of 128 bytes per row, by a producer
//     warp of their own.  Groups of four warps expand K blocks in turn: a thread owns one weight
//     row, reads its 64 codes, converts them to fp16 (int8 codes are exact, the row scale is applied
//     in the epilogue; a Q4 weight becomes fp16(code * block scale)) and stores them to TENSOR
//     memory, from where the MMA takes its M operand.  The expanded weights so never cross shared
//     memory: writing them there and reading them back cost more shared-memory bandwidth (2 x 16 KB
//     per K block) than everything else together, and set the pace of the packed formats.
//   * few tiles (a per-layer projection of a prompt): the K blocks of a tile are split over a
//     cluster of 2..8 blocks, whose fp32 partial sums meet through distributed shared memory, each
//     block finishing its share of the tokens; the sums are added in rank order.
//   * long calls: two blocks of a cluster share a tile of 256 rows (cta_group::2), each with its half of the rows and of the
//     tokens; one of them issues the MMAs of both.
//   * every block walks K from a starting place of its own, so that the blocks do not all ask for
//     the same lines of the token operand at the same moment.
#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cstring>
#include <memory>
#include <type_traits>

#include "kernels.h"
#include "plan.h"
#include "ptx.cuh"

namespace nnb {
namespace {

constexpr int BM = 128;       // weight rows per tile (UMMA M)
constexpr int BK = 64;        // K elements per block = one 128-byte swizzle span of fp16
constexpr int A_BYTES = BM * BK * 2;  // 16 KB
constexpr int RAW_BYTES = BM * 128;   // packed span of one weight: 128 bytes of each of the tile's rows
constexpr int SC_BYTES = BM * 16;     // Q4: the block scales of a span
constexpr int RING_MAX = 16;          // token (and fp16 weight) stages
constexpr int RAW_MAX = 8;            // packed spans
constexpr int SLAB_MAX = 128;         // tokens per output slab (a staging buffer of 128 x 128 fp16 = 32 KB)
constexpr int SMEM_LIMIT = 227 * 1024;
// K blocks per packed span, and as many groups of four expanding warps
__host__ __device__ constexpr int span_blocks(int wfmt) { return wfmt == FMT_Q4 ? 4 : wfmt == FMT_INT8 ? 2 : 1; }
__host__ __device__ constexpr int dq_warps(int wfmt) { return wfmt == FMT_FP16 ? 0 : 4 * span_blocks(wfmt); }
// epilogue warps: one or two groups of four, which take the 16-token steps of a slab in turn (Q4: the expanding warps leave
// registers for four)
__host__ __device__ constexpr int epi_warps(int wfmt) { return wfmt == FMT_Q4 ? 4 : 8; }
__host__ __device__ constexpr int raw_stage_bytes(int wfmt) { return RAW_BYTES + (wfmt == FMT_Q4 ? SC_BYTES : 0); }
__host__ __device__ constexpr int gemm_threads(int wfmt) {
    return (2 + epi_warps(wfmt)) * 32 + (wfmt == FMT_FP16 ? 0 : dq_warps(wfmt) * 32 + 32);
}

// shared-memory header: barriers and the tensor-memory address
constexpr int H_FULL = 0, H_EMPTY = H_FULL + RING_MAX * 8, H_RAW_FULL = H_EMPTY + RING_MAX * 8, H_RAW_EMPTY = H_RAW_FULL + RAW_MAX * 8;
constexpr int H_ACC_FULL = H_RAW_EMPTY + RAW_MAX * 8, H_ACC_EMPTY = H_ACC_FULL + 16, H_RES = H_ACC_EMPTY + 16, H_TMEM = H_RES + 8, H_XCHG = H_TMEM + 8;
constexpr int HDR = 1024;
constexpr int SWAP_BYTES = 8192;   // the SwiGLU epilogue's two exchange buffers (16 tokens x 64 rows fp32 each) of four warps, behind the output slabs
static_assert(H_XCHG + 8 <= HDR, "header");

// The maps travel in a parameter of their own: their address is taken, and a scalar beside them would be read
// through generic loads.
struct GemmMaps {
    alignas(64) CUtensorMap w[3];    // weights: fp16 [N][K] half, box 64 x 128; packed: bytes, box 128 B x 128 (128-byte swizzle);
                                     // one per segment.  SwiGLU: [0] gate, [1] up, boxes of 64 rows
    alignas(64) CUtensorMap x;       // [M][K] fp16, box 64 x bn
    alignas(64) CUtensorMap sc[3];   // Q4 block scales, box 16 B x 128 (64) rows (one packed span), same order as w
    alignas(64) CUtensorMap out[3];  // [M][ld] fp16, box 128 (64) x slab (dense), when tma_store
};
struct GemmSeg {
    const uint16_t* scale;  // int8: row scales; Q4: block scales, [N][K / 32]
    const uint16_t* bias;
    uint16_t* out;          // [M][ld]
    int N, ld;
    int tile0;              // first row tile of the segment
};
struct GemmArgs {
    GemmSeg seg[3];
    const uint16_t* scale2;  // SwiGLU: scales of the up weight
    int nseg, M, K;
    int rows;                // output columns per tile: 128, SwiGLU 64
    int bn, ntok;            // tokens per tile, token tiles
    int tiles;               // row tile * ntok + token tile
    int ksplit, fin;         // blocks of a cluster that share a tile's K, and how many of them finish tokens
    int stages, raw_stages;
    int kps, lag;            // packed weights: K blocks per token stage; spans whose expanded blocks are in tensor memory at a time
    int accw, nacc;          // tensor-memory columns of one accumulator, and how many sets
    int tmem_cols;
    int slab, two_slabs;     // tokens per output slab; whether there are two staging buffers
    int scale_tma;           // Q4: the block scales arrive with the packed spans (else the expanding threads load them)
    int swap_off;            // SwiGLU: the exchange buffers, from the ring's start
    int xchg_off;            // split tiles: where the other blocks' parts land, from the ring's start
    int epi, tma_store, evict_first;
    int* status;
    uint16_t* peer_out[7];   // the same output block in the other ranks' gather buffers
    int npeer;
    GatherSignal sig;        // completion signal of the gather (world == 0: none)
};

// ---- tcgen05 wrappers (DUO: the forms for two blocks, cta_group::2) -------------------------
template <bool DUO>
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    if (DUO) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <bool DUO>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    if (DUO) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
template <bool DUO>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if (DUO)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
// the M operand from tensor memory: lane = row, one 32-bit column = two consecutive k
template <bool DUO>
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if (DUO)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
// (DUO: arrives on the barrier at this place in both blocks)
template <bool DUO>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    if (DUO) asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
    else asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// (the registers are valid after tmem_wait_ld, which "writes" them too so that no use moves before it)
__device__ __forceinline__ void tmem_ld16_begin(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    tmem_ld16_begin(taddr, r);
    tmem_wait_ld(r);
}
// 16 columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- tensor store (shared -> global) ------------------------------------------------------
__device__ __forceinline__ void tma_store_2d(const void* tmap, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(src), "r"(x), "r"(y)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- cluster ------------------------------------------------------------------------------
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Arrival on a barrier of any block of the cluster (an address from peer_smem).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <bool DUO>
__device__ __forceinline__ void arrive_on(uint32_t bar) {
    if (DUO) mbar_arrive_cluster(bar);
    else mbar_arrive(bar);
}
// An operand copy: into this block's memory, counted on `bar` (DUO: a barrier of either block).
template <bool DUO>
__device__ __forceinline__ void load_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar, uint64_t policy) {
    if (!DUO) return tma_load_2d(dst, tmap, x, y, bar, policy);
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(bar), "l"(policy)
        : "memory");
}
// Shared memory of this block -> shared memory of another block of the cluster, counted on that block's barrier.
__device__ __forceinline__ void bulk_s2peer(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Shared-memory matrix descriptor, K-major operand in 128-byte-swizzled rows of 128 bytes: start address >> 4,
// stride between 8-row groups = 1024 bytes, descriptor version 1, layout type 2 (128-byte swizzle); the leading
// offset is not used by this layout.  The high word never changes, the low word is the 16-byte address (14 bits) plus
// the constant leading-offset field, so a K step of 32 bytes inside a swizzle span is "+ 2" on the low word.
constexpr uint32_t DESC_HI = (uint32_t)((1024 >> 4) & 0x3FFF) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }
__device__ __forceinline__ uint64_t desc_of(uint32_t lo) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(DESC_HI));
    return d;
}
// Instruction descriptor: fp32 accumulate, fp16 x fp16, both operands K-major, M = 128 (two blocks: 256), N = bn.
__device__ __forceinline__ uint32_t instr_desc_f16(int bn, int m) {
    return (1u << 4) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// One lane of a convergent warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// Whether any epilogue thread's flag is set.
template <int EPI_WARPS>
__device__ __forceinline__ bool epilogue_any(bool f) {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 3, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((int)f), "n"(EPI_WARPS * 32) : "memory");
    return r != 0;
}

// Rows [m, m + rows) x columns [n0, n0 + cols) of a [.][ld] fp16 matrix of N columns, between global memory and a dense slab of
// `cols` columns in shared memory, by the epilogue threads: a warp takes a row, two values per lane and step where the
// rows are 4-byte aligned.  (One 2-byte store per value straight from the accumulator's lanes took 140 clocks per token.)
template <bool IN, int EPI_WARPS>
__device__ __forceinline__ void copy_rows(uint16_t* out, int ld, int N, int n0, int m, int rows, int cols, uint32_t slab, int et) {
    const int lane = et & 31, valid = min(cols, N - n0);
    const bool pairs = ((ld | n0) & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0;
    for (int r = et >> 5; r < rows; r += EPI_WARPS) {
        uint16_t* dst = out + (size_t)(m + r) * ld + n0;
        const uint32_t src = slab + (uint32_t)(r * cols * 2);
        if (pairs) {
            for (int c = lane * 2; c < valid; c += 64) {
                if (c + 1 < valid) {
                    uint32_t v;
                    if (IN) {
                        v = *reinterpret_cast<const uint32_t*>(dst + c);
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(src + c * 2), "r"(v) : "memory");
                    } else {
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(src + c * 2) : "memory");
                        *reinterpret_cast<uint32_t*>(dst + c) = v;
                    }
                } else if (IN) {
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(src + c * 2), "h"(dst[c]) : "memory");
                } else {
                    uint16_t v;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(src + c * 2) : "memory");
                    dst[c] = v;
                }
            }
        } else {
#pragma unroll 4
            for (int c = lane; c < valid; c += 32) {
                uint16_t v;
                if (IN) {
                    v = dst[c];
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(src + c * 2), "h"(v) : "memory");
                } else {
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(src + c * 2) : "memory");
                    dst[c] = v;
                }
            }
        }
    }
}

// Position in a ring of `n` slots: slot number and the parity of the pass, stepped instead of divided out.
struct RingPos {
    int s = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void next(int n) { advance(1, n); }
    __device__ __forceinline__ void advance(int k, int n) {   // 0 <= k <= n
        s += k;
        if (s >= n) {
            s -= n;
            ph ^= 1u;
        }
    }
};

// Long wait of an epilogue warp (a whole K loop): one lane looks every hundred nanoseconds or so; bounded, the same answer in
// every lane.
__device__ __forceinline__ bool wait_asleep(uint32_t bar, uint32_t parity) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) {
        const long long t0 = clock64();
        while (!mbar_try_wait(bar, parity)) {
            __nanosleep(100);
            if (clock64() - t0 > WAIT_CYCLES) {
                ok = 0;
                break;
            }
        }
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// Wait of a whole warp: the hardware parks it (a warp that polls takes issue slots from the ones that convert), bounded like
// mbar_wait_bounded; the same answer in every lane.
__device__ __forceinline__ bool wait_parked(uint32_t bar, uint32_t parity) {
    bool ok = mbar_try_wait(bar, parity) != 0;
    if (!ok) {
        const long long t0 = clock64();
        do {
            uint32_t done;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done) : "r"(bar), "r"(parity), "r"(1000000u) : "memory");
            ok = done != 0;
        } while (!ok && clock64() - t0 < WAIT_CYCLES);
    }
    return __all_sync(0xffffffffu, ok) != 0;
}

// Eight 4-bit codes of one word -> four registers of two fp16 each, in k order, times the block's scale: fp16(code * scale).
// A byte holds two consecutive codes; it is copied to both halves of a register, of which the low one keeps its low nibble
// (mantissa bits 0..3 of 1024.0h) and the high one its high nibble (bits 4..7 of 64.0h); both offsets come off exactly.
__device__ __forceinline__ void expand_q4_word(uint32_t w, __half2 scale, uint32_t* o) {
    const __half2 off = __halves2half2(__ushort_as_half(0x6408), __ushort_as_half(0x5480));  // 1024 + 8, 64 + 8
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t b = __byte_perm(w, 0u, j * 0x1111u);
        uint32_t v;
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(b), "r"(0x00F0000Fu), "r"(0x54006400u));
        const __half2 h = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&v), off), scale);
        o[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
}

// x / (1 + exp(-x)) with the division's rounding: a quotient by the approximate reciprocal (1 ulp), corrected by its remainder, which
// the fused multiply-add gives exactly (P. Markstein, IBM J. Res. Dev. 34, 1990).  Outside (-86, 32) the first quotient
// stays: x itself above, where the denominator is 1, and below it less than 2^-117, -0 at the end, NaN for -inf.  For no fp32 x does it
// differ from the division where that is 1e-30 or more; the two-ulp __fdividef differs for 1.1e8 of them, which shows in fp16
// results, and is 0 to 0.2 us per call faster.  The division itself took a 512-token prompt (24 layers with gate and up of
// 4864 x 896, fp16) from 1.28 to 1.41 ms.
__device__ __forceinline__ float silu(float x) {
    const float d = 1.0f + expf(-x);
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(d));
    const float q = x * y, r = fmaf(fmaf(-q, d, x), y, q);
    return fabsf(x + 27.0f) < 59.0f ? r : q;
}

// DUO: two blocks of a cluster work on two neighbouring row tiles and the same tokens: see `duo` in gemm_choose.
template <int WFMT, bool DUO>
__global__ void __launch_bounds__(gemm_threads(WFMT), 1) linear_gemm_tc_kernel(const __grid_constant__ GemmMaps mp, const GemmArgs g) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr bool PACKED = WFMT != FMT_FP16;
    constexpr int SPAN = span_blocks(WFMT), DQ = dq_warps(WFMT), EPI_WARPS = epi_warps(WFMT), GROUPS = EPI_WARPS / 4;
    // (the shuffle tells the compiler that a warp's number is uniform, and so the control flow that depends on it)
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t s_base = smem_u32(smem);
    const uint32_t full0 = s_base + H_FULL, empty0 = s_base + H_EMPTY, raw_full0 = s_base + H_RAW_FULL, raw_empty0 = s_base + H_RAW_EMPTY;
    const uint32_t acc_full0 = s_base + H_ACC_FULL, acc_empty0 = s_base + H_ACC_EMPTY;
    const uint32_t res_bar = s_base + H_RES, xchg_bar = s_base + H_XCHG;
    const uint32_t ring = (s_base + (uint32_t)HDR + 1023u) & ~1023u;
    const int bn = g.bn, stages = g.stages, raw_stages = g.raw_stages, ntok = g.ntok, S = DUO ? 1 : g.ksplit, nacc = g.nacc, accw = g.accw;
    // Scalars used in loops are read from the parameter block once: a store the compiler cannot see through would otherwise
    // have every later use read it again.
    const bool pair = g.epi == EPI_SWIGLU;   // a tile is 64 rows of each of two weights
    const int trows = g.rows;
    const int epi = g.epi, slab = g.slab, gM = g.M, npeer = g.npeer, tile_end = g.tiles;
    const int lag = g.lag;   // packed weights: spans whose expanded blocks are in tensor memory at a time (1, 2 or 4)
    const bool tma_store = g.tma_store != 0;
    int* const status = g.status;
    const int half_rank = DUO ? (int)(blockIdx.x & 1u) : 0;            // 0: the block that issues the MMAs of both
    const int xtok = DUO ? bn / 2 : bn;                                // tokens that this block loads
    const int b_bytes = xtok * BK * 2;                                 // a multiple of 2 KB
    // K blocks per stage: one; packed weights: 1, 2 or 4 (dividing the span's), so that few waits and commits are paid per block
    const int kps = PACKED ? g.kps : 1;
    const int b_off = PACKED ? 0 : A_BYTES, stage_bytes = b_off + kps * b_bytes;
    const uint32_t raw_ring = ring + (uint32_t)(stages * stage_bytes);
    constexpr int RAW_STAGE = raw_stage_bytes(WFMT);
    const uint32_t out_stage = raw_ring + (PACKED ? (uint32_t)(raw_stages * RAW_STAGE) : 0u);
    const uint32_t xchg = ring + (uint32_t)g.xchg_off, swap_base = ring + (uint32_t)g.swap_off;
    // this block's share of K, in units of one K block (fp16) or one packed span
    const int nkb = (g.K + BK - 1) / BK, nunits = (nkb + SPAN - 1) / SPAN;
    const int rank = S > 1 ? (int)(blockIdx.x % (unsigned)S) : 0;
    const int u0 = rank * nunits / S, nu = (rank + 1) * nunits / S - u0;
    const int tile_first = DUO ? (int)(blockIdx.x >> 1) : S > 1 ? (int)(blockIdx.x / (unsigned)S) : (int)blockIdx.x;
    const int fin = g.fin, cps = bn / fin;                              // blocks of a cluster that finish tokens, and how many each
    const int tile_step = DUO ? (int)(gridDim.x >> 1) : S > 1 ? g.tiles : (int)gridDim.x;   // a split tile: one per cluster
    // DUO: a tile number stands for two row tiles.  The second one of the last pair may lie past the end: its copies bring zeros.
    auto row_tile = [&](int tile) { return DUO ? 2 * (tile / ntok) + half_rank : tile / ntok; };
    auto segment = [&](int rt) { return (g.nseg > 2 && rt >= g.seg[2].tile0) ? 2 : (g.nseg > 1 && rt >= g.seg[1].tile0) ? 1 : 0; };
    auto seg_at = [&](int si) { return si == 0 ? g.seg[0] : si == 1 ? g.seg[1] : g.seg[2]; };
    auto first_unit = [&](int tile) { return (int)((unsigned)(tile / ntok * 7) % (unsigned)nu); };   // where the walk over K starts

    // one barrier per thread: a single thread took a thousand clocks over them
    if (tid < RING_MAX) {
        if (tid < stages) mbar_init(full0 + tid * 8, PACKED ? 1 + 4 * kps * (DUO ? 2 : 1) : 1);   // the copies (and the four warps that expand each K block)
    } else if (tid < 2 * RING_MAX) {
        if (tid - RING_MAX < stages) mbar_init(empty0 + (tid - RING_MAX) * 8, 1);
    } else if (tid < 2 * RING_MAX + 4) {
        const int a = tid - 2 * RING_MAX;
        mbar_init((a < 2 ? acc_full0 : acc_empty0) + (a & 1) * 8, a < 2 ? 1 : EPI_WARPS * (DUO ? 2 : 1));
    } else if (tid == 2 * RING_MAX + 4) {
        mbar_init(res_bar, 1);
    } else if (tid == 2 * RING_MAX + 5) {
        mbar_init(xchg_bar, 1);
        if (S > 1 && rank < fin) mbar_arrive_expect_tx(xchg_bar, (uint32_t)((S - 1) * cps * BM * 4));
    } else if (PACKED && tid >= 64 && tid < 64 + 2 * RAW_MAX) {
        const int r = (tid - 64) & (RAW_MAX - 1);
        if (r < raw_stages) mbar_init((tid < 64 + RAW_MAX ? raw_full0 : raw_empty0) + r * 8, tid < 64 + RAW_MAX ? 1 : DQ);
    }
    mbar_init_fence();
    if (warp == 1) tmem_alloc<DUO>(s_base + H_TMEM, (uint32_t)g.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + H_TMEM);
    if (DUO) {   // both blocks hold their tensor memory and their barriers are ready
        cluster_arrive();
        cluster_wait();
    }
    // where operands and expanded blocks are announced, and accumulators given back: the issuing block
    const uint32_t full_at = DUO ? peer_smem(full0, 0) : full0, acc_empty_at = DUO ? peer_smem(acc_empty0, 0) : acc_empty0;
    const uint32_t at_base = tmem_base + (uint32_t)(nacc * accw);
    // The launch after this one may begin (its prologue, and weights that no launch writes) once every block of this one
    // holds its tensor memory: a later block must never take columns that an earlier launch still has to get.
    if (tid == 0) pdl_launch_dependents();
    if (S > 1) {   // the other blocks' memory may be written once they run: their arrivals are awaited before anything is sent
        __syncwarp();
        cluster_arrive();
    }

    // ---- the finish of a tile, by the epilogue warps: columns [col0, col0 + ncols) of the accumulators at `acc_col` ----
    const int q = warp & 3, group = (warp - 2) >> 2 & 1;
    int n_slabs = 0;
    const bool inplace = epi == EPI_RESIDUAL || epi == EPI_SILU_GATE;
    constexpr int CH = 16;   // columns read at a time
    const bool two_slabs = DUO && !PACKED && g.two_slabs;
    const uint32_t stage_step = two_slabs ? (uint32_t)((slab + 15) / 16 * 16 * trows * 2) : 0u;
    auto stage_of = [&](int n) { return out_stage + (uint32_t)(n & 1) * stage_step; };
    auto prefetch_slab = [&](int tile, int col) {   // in-place epilogues: the values to be updated, into the next staging buffer
        const int rt = row_tile(tile), tt = tile % ntok, si = segment(rt);
        if (warp == 2 && lane == 0) {
            if (!two_slabs && n_slabs > 0) bulk_wait_read0();
            mbar_arrive_expect_tx(res_bar, (uint32_t)(slab * BM * 2));   // (SwiGLU is not in place: tiles of 128 rows here)
            tma_load_2d(stage_of(n_slabs), &mp.out[si], (rt - seg_at(si).tile0) * BM, tt * bn + col, res_bar, l2_policy_evict_normal());
        }
    };
    auto finish_tile = [&](int tile, uint32_t acc_col, int col0, int ncols, bool& failed, uint32_t ready_bar, uint32_t ready_ph, uint32_t release_bar) __attribute__((always_inline)) {
        const int rt = row_tile(tile), tt = tile % ntok, si = segment(rt);
        const GemmSeg sg = seg_at(si);
        // row: this thread's accumulator lane; orow: the output column (within the tile) it finishes
        const int n0 = (rt - sg.tile0) * trows, row = q * 32 + lane, orow = pair ? row & 63 : row, n = n0 + orow, m0 = tt * bn;
        const bool row_ok = n < sg.N;
        float rs = 1.f, bias = 0.f;
        if (WFMT == FMT_INT8 && row_ok) rs = __half2float(__ushort_as_half((pair && row >= 64 ? g.scale2 : sg.scale)[n]));
        const bool biased = sg.bias != nullptr;
        if (biased && row_ok) bias = __half2float(__ushort_as_half(sg.bias[n]));
        if (ready_bar) {   // (the scale and the bias are on their way by now)
            if (!failed && !wait_asleep(ready_bar, ready_ph)) {
                failed = true;
                if (lane == 0) *reinterpret_cast<volatile int*>(status) = 5;
            }
            failed = epilogue_any<EPI_WARPS>(failed);   // (the warps meet at barriers below: all of them take the same way)
            tc_fence_after();
        }
        const uint32_t tm = tmem_base + acc_col + ((uint32_t)(q * 32) << 16);
        // the accumulator is free as soon as this warp's last columns have been read
        bool released = release_bar == 0u;
        auto release = [&]() {
            released = true;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_on<DUO>(release_bar);
        };
        // the sums of columns c .. c + CH - 1 (a split tile: all ranks' parts, in rank order), times the int8 row scale, from the
        // accumulator's columns in r
        auto sums = [&](int c, const uint32_t (&r)[CH], float (&v)[CH]) __attribute__((always_inline)) {
#pragma unroll
            for (int j = 0; j < CH; ++j) v[j] = __uint_as_float(r[j]);
            if (S > 1) {
                float t[CH];
#pragma unroll
                for (int j = 0; j < CH; ++j) t[j] = 0.f;
                for (int p = 0; p < S; ++p) {
                    if (p == rank) {
#pragma unroll
                        for (int j = 0; j < CH; ++j) t[j] += v[j];
                        continue;
                    }
                    const uint32_t src = xchg + (uint32_t)((((p < rank ? p : p - 1) * (cps / 4) + (c - col0) / 4) * BM + row) * 16);
                    float o[CH];
#pragma unroll
                    for (int j = 0; j < CH; j += 4)
                        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(o[j]), "=f"(o[j + 1]), "=f"(o[j + 2]), "=f"(o[j + 3]) : "r"(src + (uint32_t)(j / 4 * BM * 16)));
#pragma unroll
                    for (int j = 0; j < CH; ++j) t[j] += o[j];
                }
#pragma unroll
                for (int j = 0; j < CH; ++j) v[j] = t[j];
            }
            if (WFMT == FMT_INT8) {
#pragma unroll
                for (int j = 0; j < CH; ++j) v[j] *= rs;
            }
        };
        // SwiGLU: the gate row's thread finishes the first half of the columns, the up row's thread the second; each hands the
        // other its values of the other half through shared memory (two buffers in turn, so one barrier per CH columns).
        int swaps = 0;
        auto swap_halves = [&](float (&v)[CH]) __attribute__((always_inline)) {
            const int up = row >> 6;
            const uint32_t buf = swap_base + (uint32_t)(group * SWAP_BYTES + (swaps++ & 1) * 4096), at = buf + (uint32_t)(orow * 16);
            const uint32_t mine = at + (uint32_t)(up * 2048), theirs = at + (uint32_t)((up ^ 1) * 2048);
#pragma unroll
            for (int j = 0; j < CH / 2; j += 4) {
                const float a = up ? v[j] : v[CH / 2 + j], b = up ? v[j + 1] : v[CH / 2 + j + 1];
                const float c = up ? v[j + 2] : v[CH / 2 + j + 2], d = up ? v[j + 3] : v[CH / 2 + j + 3];
                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(mine + (uint32_t)(j / 4 * 1024)), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
            }
            asm volatile("bar.sync %0, 128;" ::"r"(4 + group) : "memory");
#pragma unroll
            for (int j = 0; j < CH / 2; j += 4) {
                float o[4];
                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "r"(theirs + (uint32_t)(j / 4 * 1024)) : "memory");
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float gt = up ? o[i] : v[j + i], u = up ? v[CH / 2 + j + i] : o[i];
                    v[j + i] = silu(gt) * u;
                }
            }
        };
        // The mode (0: store; 1: bias; 2: residual; 3: SiLU gate; 4: SwiGLU) is a compile-time value of the column loops: a
        // uniform branch per value would cost several times the value's arithmetic.
        auto value = [&](auto mode, float v, uint16_t prev) {
            constexpr int MODE = decltype(mode)::value;
            if (MODE == 1) v = __fadd_rn(__half2float(__float2half_rn(v)), bias);   // added to the rounded result, as bias_add_rowmajor does
            if (MODE == 2) v = __half2float(__ushort_as_half(prev)) + v;
            if (MODE == 3) {
                const float gt = __half2float(__ushort_as_half(prev));
                v = (gt / (1.0f + expf(-gt))) * v;
            }
            return v;
        };
        auto by_mode = [&](auto&& f) {
            if (epi == EPI_RESIDUAL) f(std::integral_constant<int, 2>{});
            else if (epi == EPI_SILU_GATE) f(std::integral_constant<int, 3>{});
            else if (pair) f(std::integral_constant<int, 4>{});
            else if (biased) f(std::integral_constant<int, 1>{});
            else f(std::integral_constant<int, 0>{});
        };
        if (!failed) {
            // Lay the tile out as [token][output column] in shared memory and let one tensor store per slab write it; the tensor
            // map clips the rows and columns past M and N.  (Outputs whose rows are not 16-byte aligned: the warps copy the slab out
            // row by row, and for the in-place forms in.)  Two columns of one token per 32-bit store: neighbouring lanes swap
            // halves, the even lane then holds token j of both columns and the odd lane token j + 1.
            const uint32_t pick = (lane & 1) ? 0x3276u : 0x5410u, pitch = (uint32_t)(trows * 2);
            // The next columns are on their way out of tensor memory while these are finished.
            uint32_t r[CH];
            constexpr bool AHEAD = WFMT != FMT_Q4;   // (Q4's epilogue has no registers left for it)
            if (AHEAD && group * CH < slab) tmem_ld16_begin(tm + (uint32_t)(col0 + group * CH), r);
            for (int h0 = 0; h0 < ncols; h0 += slab) {
                const int hrows = min(slab, ncols - h0);
                if (!tma_store) {
                    asm volatile("bar.sync 2, %0;" ::"n"(EPI_WARPS * 32) : "memory");   // the previous slab has been copied out
                    if (inplace) {
                        copy_rows<true, EPI_WARPS>(sg.out, sg.ld, sg.N, n0, m0 + col0 + h0, min(hrows, gM - m0 - col0 - h0), trows, out_stage, tid - 64);
                        asm volatile("bar.sync 2, %0;" ::"n"(EPI_WARPS * 32) : "memory");
                    }
                } else if (inplace) {
                    if (!mbar_wait_bounded_warp(res_bar, (uint32_t)(n_slabs & 1))) {
                        failed = true;
                        if (lane == 0) *reinterpret_cast<volatile int*>(status) = 9;
                    }
                } else if (!two_slabs && n_slabs > 0) {
                    // the previous slab's store must have finished reading the staging buffer
                    if (warp == 2 && lane == 0) bulk_wait_read0();
                    asm volatile("bar.sync 2, %0;" ::"n"(EPI_WARPS * 32) : "memory");
                }
                const uint32_t buf = tma_store ? stage_of(n_slabs) : out_stage;
                const uint32_t pair0 = buf + (uint32_t)((orow & ~1) * 2) + (lane & 1) * pitch, mine0 = buf + (uint32_t)(orow * 2);
                // (a slab's last columns may be fewer than CH: the buffer has room for the rest, which no store reads)
                by_mode([&](auto mode) __attribute__((always_inline)) {
                    constexpr int MODE = decltype(mode)::value, NC = MODE == 4 ? CH / 2 : CH;
                    const int half = MODE == 4 && row >= 64 ? CH / 2 : 0;
                    for (int c = group * CH; c < hrows; c += GROUPS * CH) {
                        float v[CH];
                        if (AHEAD) tmem_wait_ld(r);
                        else tmem_ld16(tm + (uint32_t)(col0 + h0 + c), r);
                        sums(col0 + h0 + c, r, v);
                        const int after = c + GROUPS * CH < hrows ? h0 + c + GROUPS * CH : h0 + slab + group * CH;
                        if (after >= ncols) {
                            if (!released) release();
                        } else if (AHEAD) {
                            tmem_ld16_begin(tm + (uint32_t)(col0 + after), r);
                        }
                        if (MODE == 4) swap_halves(v);
                        const uint32_t off = (uint32_t)(c + half) * pitch;
                        uint16_t old[CH];
                        if (MODE == 2 || MODE == 3) {
#pragma unroll
                            for (int j = 0; j < CH; ++j)
                                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(old[j]) : "r"(mine0 + off + (uint32_t)(j * (BM * 2))) : "memory");
                            __syncwarp();   // the neighbour writes where this lane has read
                        }
                        // (all exchanges before the first store: one at a time, a value pair takes the latency of its exchange)
                        uint32_t own[NC / 2], other[NC / 2];
#pragma unroll
                        for (int j = 0; j < NC; j += 2) {
                            const __half2 h2 = __floats2half2_rn(value(mode, v[j], MODE == 2 || MODE == 3 ? old[j] : (uint16_t)0),
                                                                 value(mode, v[j + 1], MODE == 2 || MODE == 3 ? old[j + 1] : (uint16_t)0));
                            own[j / 2] = *reinterpret_cast<const uint32_t*>(&h2);
                        }
#pragma unroll
                        for (int j = 0; j < NC / 2; ++j) other[j] = __shfl_xor_sync(0xffffffffu, own[j], 1);
#pragma unroll
                        for (int j = 0; j < NC; j += 2)
                            asm volatile("st.shared.u32 [%0], %1;" ::"r"(pair0 + off + (uint32_t)j * (MODE == 4 ? 128u : 256u)), "r"(__byte_perm(own[j / 2], other[j / 2], pick)) : "memory");
                    }
                });
                fence_async_smem();
                // two buffers: the store before this one has read its own, which past the barrier is the next slab's
                if (two_slabs && warp == 2 && lane == 0) bulk_wait_read0();
                asm volatile("bar.sync 2, %0;" ::"n"(EPI_WARPS * 32) : "memory");
                const int rows_out = min(hrows, gM - m0 - col0 - h0);
                if (!tma_store) {
                    copy_rows<false, EPI_WARPS>(sg.out, sg.ld, sg.N, n0, m0 + col0 + h0, rows_out, trows, out_stage, tid - 64);
                    for (int p = 0; p < npeer; ++p) copy_rows<false, EPI_WARPS>(g.peer_out[p], sg.ld, sg.N, n0, m0 + col0 + h0, rows_out, trows, out_stage, tid - 64);
                    continue;
                }
                if (warp == 2 && lane == 0 && (!DUO || n0 < sg.N)) tma_store_2d(&mp.out[si], buf, n0, m0 + col0 + h0);
                ++n_slabs;
                if (inplace && h0 + slab < ncols) prefetch_slab(tile, col0 + h0 + slab);   // (the first slab of a tile was asked for at its start)
                if (npeer > 0) {
                    // peers get the slab in 16-byte pieces, 256 contiguous bytes per token row (a plain store: tiles of 128 columns)
                    const int et = (warp - 2) * 32 + lane;
                    for (int i = et; i < rows_out * 16; i += EPI_WARPS * 32) {
                        const int mr = i >> 4, ch = i & 15;
                        if (n0 + ch * 8 >= sg.N) continue;
                        uint4 v;
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                     : "r"(buf + (uint32_t)(mr * (BM * 2) + ch * 16)) : "memory");
                        const size_t o = (size_t)(m0 + col0 + h0 + mr) * sg.ld + n0 + ch * 8;
#pragma unroll
                        for (int p = 0; p < 7; ++p)
                            if (p < npeer) *reinterpret_cast<uint4*>(g.peer_out[p] + o) = v;
                    }
                }
            }
        }
        if (!released) release();
    };

    bool failed = false;
    // The producers and the MMA issuer walk their loops as whole warps and elect one lane where something is issued: addresses,
    // descriptors and coordinates then are warp-uniform values in uniform registers, which the copy and MMA instructions take
    // directly.  (A single lane under "lane == 0" spent 500-700 clocks per K block on the issuing side alone, twice what the
    // tensor core needs for 128 x 256 x 64; whole-warp loops with one barrier and one commit per K block, as below, do not.)
    if (warp == 0) {
        // ---- TMA producer: walks (tile, K block) and keeps the ring full ----
        const uint64_t policy = l2_policy_evict_normal();
        int ahead = 0;
        if (!PACKED && tile_first < tile_end) {
            // fp16 weights of the ring's first pass: they do not depend on the launch before this one
            const int rt = row_tile(tile_first), f = first_unit(tile_first), si = segment(rt), row0 = (rt - seg_at(si).tile0) * trows;
            ahead = min(stages, nu);
            if (elect_one()) {
                for (int j = 0; j < ahead; ++j) {
                    const int kb = u0 + (f + j < nu ? f + j : f + j - nu);
                    if (half_rank == 0) mbar_arrive_expect_tx(full0 + j * 8, (uint32_t)(stage_bytes * (DUO ? 2 : 1)));   // both blocks' copies
                    load_2d<DUO>(ring + j * stage_bytes, &mp.w[si], kb * BK, row0, full_at + j * 8, policy);
                    if (pair) load_2d<DUO>(ring + j * stage_bytes + A_BYTES / 2, &mp.w[1], kb * BK, row0, full_at + j * 8, policy);
                }
            }
            __syncwarp();
        }
        pdl_wait_prior_grid();
        RingPos r;
        int it = 0;
        bool ok = true;
        for (int tile = tile_first; tile < tile_end && ok; tile += tile_step) {
            const int rt = row_tile(tile), x0 = tile % ntok * bn + half_rank * xtok, si = segment(rt), row0 = (rt - seg_at(si).tile0) * trows;
            const CUtensorMap* const mw = &mp.w[si];
            int u = first_unit(tile);
            for (int j = 0; j < nu && ok; ++j, u = (u + 1 == nu ? 0 : u + 1)) {
                const int kb0 = (u0 + u) * SPAN, nb = min(SPAN, nkb - kb0);
                for (int p = 0; p < nb; p += kps, ++it, r.next(stages)) {   // (kps divides SPAN: a stage never crosses a span)
                    if (it >= stages && !wait_parked(empty0 + r.s * 8, r.ph ^ 1u)) {
                        if (lane == 0) *reinterpret_cast<volatile int*>(status) = 3;
                        ok = false;
                        break;
                    }
                    if (elect_one()) {
                        const uint32_t dst = ring + r.s * stage_bytes, own = full0 + r.s * 8, bar = full_at + r.s * 8;
                        if (PACKED) {
                            const int n = min(kps, nb - p);
                            if (half_rank == 0) mbar_arrive_expect_tx(own, (uint32_t)(n * b_bytes * (DUO ? 2 : 1)));
                            for (int i = 0; i < n; ++i) load_2d<DUO>(dst + i * b_bytes, &mp.x, (kb0 + p + i) * BK, x0, bar, policy);
                        } else {
                            if (it >= ahead) {
                                if (half_rank == 0) mbar_arrive_expect_tx(own, (uint32_t)(stage_bytes * (DUO ? 2 : 1)));
                                load_2d<DUO>(dst, mw, kb0 * BK, row0, bar, policy);
                                if (pair) load_2d<DUO>(dst + A_BYTES / 2, &mp.w[1], kb0 * BK, row0, bar, policy);
                            }
                            load_2d<DUO>(dst + b_off, &mp.x, kb0 * BK, x0, bar, policy);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint32_t idesc = instr_desc_f16(bn, DUO ? 2 * BM : BM);
        const uint32_t lo_step = (uint32_t)stage_bytes >> 4, lo0 = smem_desc_lo(ring), b_lo_off = (uint32_t)b_off >> 4, blk_step = (uint32_t)b_bytes >> 4;
        uint32_t lo = lo0, at = at_base;   // descriptor of the stage; this span's expanded blocks
        RingPos r;
        int tl = 0, nspan = 0;
        bool ok = half_rank == 0;
        for (int tile = tile_first; tile < tile_end && ok; tile += tile_step, ++tl) {
            const int acc = nacc == 2 ? (tl & 1) : 0, pass = nacc == 2 ? tl >> 1 : tl;
            if (pass >= 1 && !wait_parked(acc_empty0 + acc * 8, (uint32_t)((pass - 1) & 1))) {
                if (lane == 0) *reinterpret_cast<volatile int*>(status) = 6;
                break;
            }
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(acc * accw);
            uint32_t accumulate = 0u;
            int u = PACKED ? first_unit(tile) : 0;
            for (int j = 0; j < nu && ok; ++j) {
                const int nb = PACKED ? min(SPAN, nkb - (u0 + u) * SPAN) : 1;
                for (int p = 0; p < nb; p += kps) {
                    if (!wait_parked(full0 + r.s * 8, r.ph)) {
                        if (lane == 0) *reinterpret_cast<volatile int*>(status) = 4;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if (elect_one()) {
                        const int n = PACKED ? min(kps, nb - p) : 1;
                        for (int i = 0; i < n; ++i) {
                            const uint32_t b_lo = lo + b_lo_off + (uint32_t)i * blk_step, a_tm = at + (uint32_t)((p + i) * 32);
#pragma unroll
                            for (int k = 0; k < BK / 16; ++k) {
                                const uint32_t acc_in = (k || i) ? 1u : accumulate;
                                if (PACKED) umma_f16_ts<DUO>(tmem_d, a_tm + (uint32_t)(k * 8), desc_of(b_lo + 2 * k), idesc, acc_in);
                                else umma_f16<DUO>(tmem_d, desc_of(lo + 2 * k), desc_of(b_lo + 2 * k), idesc, acc_in);
                            }
                        }
                        umma_commit<DUO>(empty0 + r.s * 8);  // the operands are free once these MMAs have read them
                        if (j + 1 == nu && p + kps >= nb) umma_commit<DUO>(acc_full0 + acc * 8);  // this tile's accumulators are complete
                    }
                    __syncwarp();
                    accumulate = 1u;
                    r.next(stages);
                    lo = r.s == 0 ? lo0 : lo + lo_step;
                }
                if (PACKED) {
                    if (++u == nu) u = 0;
                    if (++nspan == lag) {
                        nspan = 0;
                        at = at_base;
                    } else {
                        at += SPAN * 32;
                    }
                }
            }
        }
    } else if (PACKED && warp == 2 + EPI_WARPS + DQ) {
        // ---- packed-weight producer: runs raw_stages spans ahead of the expanding warps ----
        const bool scale_tma = WFMT == FMT_Q4 && g.scale_tma;
        const uint64_t policy = g.evict_first ? l2_policy_evict_first() : l2_policy_evict_normal();
        RingPos r;
        int it = 0;
        bool ok = true;
        for (int tile = tile_first; tile < tile_end && ok; tile += tile_step) {
            const int rt = row_tile(tile), si = segment(rt), n0 = (rt - seg_at(si).tile0) * trows;
            const CUtensorMap *const mw = &mp.w[si], *const ms = &mp.sc[si];
            int u = first_unit(tile);
            for (int j = 0; j < nu; ++j, ++it, r.next(raw_stages), u = (u + 1 == nu ? 0 : u + 1)) {
                if (it >= raw_stages && !wait_parked(raw_empty0 + r.s * 8, r.ph ^ 1u)) {
                    if (lane == 0) *reinterpret_cast<volatile int*>(status) = 11;
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t dst = raw_ring + r.s * RAW_STAGE, bar = raw_full0 + r.s * 8;
                    mbar_arrive_expect_tx(bar, (uint32_t)(RAW_BYTES + (scale_tma ? SC_BYTES : 0)));
                    tma_load_2d(dst, mw, (u0 + u) * 128, n0, bar, policy);
                    if (pair) tma_load_2d(dst + RAW_BYTES / 2, &mp.w[1], (u0 + u) * 128, n0, bar, policy);
                    if (scale_tma) {
                        tma_load_2d(dst + RAW_BYTES, ms, (u0 + u) * 16, n0, bar, policy);
                        if (pair) tma_load_2d(dst + RAW_BYTES + SC_BYTES / 2, &mp.sc[1], (u0 + u) * 16, n0, bar, policy);
                    }
                }
                __syncwarp();
            }
        }
    } else if (PACKED && warp >= 2 + EPI_WARPS) {
        // ---- expanding warps: packed span -> fp16 in tensor memory.  Group p expands K block p of every span into buffer
        //      (span mod lag, p), free once the MMAs of span - lag are done, which is what the "empty" barrier of that span's
        //      token stage says; the groups' arrivals join the token copies' on the "full" barrier of the block's stage, so
        //      the issuer waits once per stage.  A group without a block in a short last span arrives all the same, and every
        //      group waits for every span, so that no phase of a barrier can be passed unseen (the waits are by parity; the
        //      ring holds at least `lag` spans). ----
        const int grp = (warp - (2 + EPI_WARPS)) >> 2, row = q * 32 + lane;
        const uint32_t rbase = (uint32_t)((row >> 3) * 1024 + (row & 7) * 128), x7 = (uint32_t)(row & 7);
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const bool scale_tma = WFMT == FMT_Q4 && g.scale_tma;
        // Q4 without a tensor view of the scales: the two block scales of K block `kb` of this thread's row
        auto load_scales = [&](int rt, int kb) {
            const GemmSeg sg = seg_at(segment(rt));
            const int n = (rt - sg.tile0) * trows + (pair ? row & 63 : row), K32 = g.K / 32;
            if (n >= sg.N) return 0u;
            const uint16_t* h = (pair && row >= 64 ? g.scale2 : sg.scale) + (size_t)n * K32 + kb * 2;
            return (uint32_t)h[0] | (kb * 2 + 1 < K32 ? (uint32_t)h[1] << 16 : 0u);
        };
        RingPos r, t;   // packed spans; token stages (of the span's first block)
        int n = 0;      // spans so far
        RingPos old[4];         // the stages this group's arrivals went to in the last spans
        uint32_t pending = 0;
        bool ok = true;
        constexpr int NP = WFMT == FMT_INT8 ? 4 : 2;   // 16-byte pieces of a row per K block
        const int kps_log = kps == 4 ? 2 : kps - 1, sub = grp >> kps_log;
        // A store to tensor memory takes some 500 clocks to complete.  With two buffers per group the arrival for a block is
        // left until the next block's codes are converted, or until this group would have to wait (for the next span, or for the
        // MMAs that free its buffer: left pending through that wait the arrival would hold up the MMAs of its own span as well).
        const bool defer = lag >= 2;
        uint32_t at = at_base + (uint32_t)(grp * 32) + lane_off, at_end = at + (uint32_t)(lag * SPAN * 32);
        const uint32_t at_first = at;
        auto flush = [&]() {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_on<DUO>(pending);
            pending = 0;
        };
        for (int tile = tile_first; tile < tile_end && ok; tile += tile_step) {
            int u = first_unit(tile);
            for (int j = 0; j < nu; ++j) {
                const uint32_t rbar = raw_full0 + r.s * 8;
                const int kb0 = (u0 + u) * SPAN, nb = min(SPAN, nkb - kb0), nsub = (nb + kps - 1) >> kps_log;
                // the stage of this group's block (or the span's last one)
                RingPos mine = t;
                mine.advance(min(sub, nsub - 1), stages);
                t.advance(nsub, stages);
                const RingPos free_at = lag == 4 ? old[3] : lag == 2 ? old[1] : old[0];
                if (pending && !__all_sync(0xffffffffu, mbar_test_wait(rbar, r.ph) != 0 && (n < lag || mbar_test_wait(empty0 + free_at.s * 8, free_at.ph) != 0)))
                    flush();
                if (!wait_parked(rbar, r.ph) || (n >= lag && !wait_parked(empty0 + free_at.s * 8, free_at.ph))) {
                    if (lane == 0) *reinterpret_cast<volatile int*>(status) = 10;
                    ok = false;
                    break;
                }
                if (grp < nb) {
                    tc_fence_after();
                    const uint32_t span = raw_ring + r.s * RAW_STAGE;
                    uint32_t c[NP][4], sc = 0u;
#pragma unroll
                    for (int i = 0; i < NP; ++i)
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(c[i][0]), "=r"(c[i][1]), "=r"(c[i][2]), "=r"(c[i][3])
                                     : "r"(span + rbase + (((uint32_t)(grp * (8 / SPAN) + i) ^ x7) << 4)));
                    if (scale_tma) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc) : "r"(span + RAW_BYTES + row * 16 + grp * 4));
                    else if (WFMT == FMT_Q4) sc = load_scales(row_tile(tile), kb0 + grp);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t o[16];
                        if (WFMT == FMT_INT8) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) int8x4_to_half2x2(c[(h * 2 + i / 4) % NP][i % 4], o[2 * i], o[2 * i + 1]);
                        } else {
                            const uint32_t sb = __byte_perm(sc, 0u, h ? 0x3232u : 0x1010u);
#pragma unroll
                            for (int i = 0; i < 4; ++i) expand_q4_word(c[h % NP][i], *reinterpret_cast<const __half2*>(&sb), o + 4 * i);
                        }
                        if (h == 0 && pending) flush();
                        tmem_st16(at + (uint32_t)(h * 16), o);
                    }
                    pending = full_at + mine.s * 8;
                    if (!defer) flush();
                } else {
                    if (pending) flush();
                    if (sub < nsub && lane == 0) arrive_on<DUO>(full_at + mine.s * 8);
                }
                if ((at += SPAN * 32) == at_end) at = at_first;
                old[3] = old[2];
                old[2] = old[1];
                old[1] = old[0];
                old[0] = mine;
                ++n;
                __syncwarp();
                if (lane == 0) mbar_arrive(raw_empty0 + r.s * 8);   // this warp is done with the span
                r.next(raw_stages);
                if (++u == nu) u = 0;
            }
        }
        if (pending) flush();
    } else {
        // ---- epilogue warps ----
        pdl_wait_prior_grid();
        int tl = 0;
        for (int tile = tile_first; tile < tile_end; tile += tile_step, ++tl) {
            const int acc = nacc == 2 ? (tl & 1) : 0, pass = nacc == 2 ? tl >> 1 : tl;
            if (inplace && tma_store && rank < fin) prefetch_slab(tile, rank * cps);
            if (S > 1) {
                if (!wait_asleep(acc_full0, 0u)) {
                    failed = true;
                    if (lane == 0) *reinterpret_cast<volatile int*>(status) = 5;
                }
                failed = epilogue_any<EPI_WARPS>(failed);
                tc_fence_after();
            } else {
                finish_tile(tile, (uint32_t)(acc * accw), 0, bn, failed, acc_full0 + acc * 8, (uint32_t)(pass & 1), acc_empty_at + acc * 8);
            }
        }
    }
    if (S > 1) {
        // Every block of the cluster holds its part of the same tile's sums; block d < fin finishes tokens [d cps, (d + 1) cps).
        // A part is laid out as [4 tokens][row][4 fp32] in the operand ring (idle once this block's MMAs are done) and crosses
        // the cluster as one bulk copy.  (Stores by the threads crossed it at 4 bytes per clock: 8 us for a 128 x 112 part.)
        const bool epi_warp = warp >= 2 && warp < 2 + EPI_WARPS;
        __syncwarp();
        cluster_wait();
        if (epi_warp) {
            const int row = q * 32 + lane;
            const uint32_t tm = tmem_base + ((uint32_t)(q * 32) << 16), part = (uint32_t)(cps * BM * 4);
            for (int d = 0; d < fin; ++d) {
                if (d == rank) continue;
                for (int c = group * CH; c < cps; c += GROUPS * CH) {
                    uint32_t r[CH];
                    tmem_ld16(tm + (uint32_t)(d * cps + c), r);
#pragma unroll
                    for (int j = 0; j < CH; j += 4)
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(ring + (uint32_t)d * part + (uint32_t)(((c + j) / 4 * BM + row) * 16)), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3])
                                     : "memory");
                }
            }
            fence_async_smem();
            asm volatile("bar.sync 2, %0;" ::"n"(EPI_WARPS * 32) : "memory");
            if (warp == 2 && elect_one()) {
                for (int dd = 1; dd <= fin; ++dd) {   // every block starts with another receiver
                    const int d = (rank + dd) % fin;
                    if (d != rank) bulk_s2peer(peer_smem(xchg, d) + (uint32_t)(rank < d ? rank : rank - 1) * part, ring + (uint32_t)d * part, part, peer_smem(xchg_bar, d));
                }
            }
            __syncwarp();
            if (rank < fin) {
                if (!wait_parked(xchg_bar, 0u)) {
                    failed = true;
                    if (lane == 0) *reinterpret_cast<volatile int*>(status) = 12;
                }
                failed = epilogue_any<EPI_WARPS>(failed);
                finish_tile(tile_first, 0u, rank * cps, cps, failed, 0u, 0u, 0u);
            }
        }
        __syncwarp();
        cluster_arrive();   // this block has its parts; awaited below, before the senders' memory goes away
    }
    if (tma_store && warp == 2 && lane == 0) bulk_wait0();  // all of this block's tensor stores have landed
    tc_fence_before();
    if (S > 1) {
        __syncwarp();
        cluster_wait();
    }
    if (DUO) {   // neither block goes while the other's MMAs, commits or arrivals may still reach it
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    __syncthreads();
    if (warp == 1) tmem_dealloc<DUO>(tmem_base, (uint32_t)g.tmem_cols);
    if (tid == 0 && g.sig.world > 0) gather_signal_block_done(g.sig);
}

// ---- launch configuration ------------------------------------------------------------------
struct GemmConfig {
    int bn, ntok, ksplit, fin;
    int stages, raw_stages, kps, lag, accw, nacc, tmem_cols, slab, two_slabs;
    int swap_off, xchg_off;
    size_t smem;
    bool duo, ok;
};

// Shared and tensor memory of one (bn, ksplit) choice.
GemmConfig gemm_geometry(int fmt, int trows, int M, int K, int bn, int ksplit, bool duo) {
    GemmConfig c = {};
    const bool packed = fmt != FMT_FP16;
    c.bn = bn;
    c.ntok = (M + bn - 1) / bn;
    c.ksplit = ksplit;
    c.duo = duo;
    c.fin = 1;
    for (int f = ksplit; f > 1; --f)
        if (bn % (16 * f) == 0) { c.fin = f; break; }
    c.accw = (bn + 31) / 32 * 32;
    const int cps = bn / c.fin;
    // One slab of up to SLAB_MAX tokens, or two halves: a slab costs its fence, barrier and store (some 800 clocks) beside 300 per
    // 16 tokens.  Two buffers, where the pace of the tensor core is otherwise the epilogue's and the ring can spare the second one.
    c.slab = cps <= SLAB_MAX ? cps : cps / 2;
    c.two_slabs = duo && !packed ? 1 : 0;
    if (ksplit > 1 && c.slab % 16 != 0) return c;   // (whole steps: the other blocks' parts end with the last token)
    // the output slab (the epilogue writes 16 tokens at a time), and what the SwiGLU epilogue swaps through
    const int slab_only = (1 + c.two_slabs) * ((c.slab + 15) / 16 * 16) * trows * 2, slab_bytes = slab_only + (trows < BM ? epi_warps(fmt) / 4 * SWAP_BYTES : 0);
    const int b_bytes = (duo ? bn / 2 : bn) * BK * 2;
    const int span = span_blocks(fmt), nkb = (K + BK - 1) / BK, units = (nkb + span - 1) / span, my_units = (units + ksplit - 1) / ksplit;
    const int room = SMEM_LIMIT - HDR - 1024 - slab_bytes;
    int stage_bytes = b_bytes + A_BYTES;
    c.kps = 1;
    if (packed) {
        // The packed spans cover the HBM latency (half of the room, as far as that is of use), the token stages that of L2.
        // As many K blocks per token stage as leave at least three stages (and two spans in all).  Whole tiles of int8
        // have the tokens of four spans: the MMAs of one, the expansion of the next and the barriers between them then overlap.
        const int rs = raw_stage_bytes(fmt);
        c.raw_stages = room / 2 / rs;
        if (c.raw_stages > RAW_MAX) c.raw_stages = RAW_MAX;
        if (ksplit > 1 && c.raw_stages > my_units) c.raw_stages = my_units;
        if (c.raw_stages < 2) c.raw_stages = 2;
        for (c.kps = span; c.kps > 1; c.kps /= 2) {
            const int n = (room - c.raw_stages * rs) / (c.kps * b_bytes);
            if (n >= 3 && n * c.kps >= 2 * span) break;
        }
        stage_bytes = c.kps * b_bytes;
        // a wide token tile: fewer spans in flight, so that the tokens of two spans fit
        while (c.raw_stages > 2 && (room - c.raw_stages * rs) / stage_bytes * c.kps < 2 * span) --c.raw_stages;
        while (ksplit == 1 && fmt == FMT_INT8 && c.raw_stages > 3 && (room - c.raw_stages * rs) / stage_bytes * c.kps < 4 * span) --c.raw_stages;
    }
    c.stages = (room - c.raw_stages * (packed ? raw_stage_bytes(fmt) : 0)) / stage_bytes;
    if (c.stages > RING_MAX) c.stages = RING_MAX;
    const int my_stages = packed ? (my_units > 2 ? my_units : 2) * span / c.kps : my_units;
    if (ksplit > 1 && c.stages > my_stages) c.stages = my_stages;
    if (c.stages < 2 || (packed && c.stages * c.kps < span)) return c;
    const size_t raws = (size_t)c.raw_stages * (packed ? raw_stage_bytes(fmt) : 0);
    if (ksplit > 1) {
        // the parts to send lie in the ring, the parts to receive behind everything else
        const size_t send = (size_t)bn * BM * 4, recv = (size_t)(ksplit - 1) * cps * BM * 4;
        const int least_stages = packed ? (2 * span / c.kps > 2 ? 2 * span / c.kps : 2) : 2;
        while (c.stages > least_stages && HDR + 1024 + (size_t)c.stages * stage_bytes + raws + slab_bytes + recv > (size_t)SMEM_LIMIT) --c.stages;
        const size_t rings = (size_t)c.stages * stage_bytes + raws;
        c.xchg_off = (int)(rings + slab_bytes);
        c.smem = HDR + 1024 + rings + slab_bytes + recv;
        if (send > rings || c.smem > (size_t)SMEM_LIMIT) return c;
        c.swap_off = (int)rings + slab_only;
    } else {
        c.swap_off = (int)((size_t)c.stages * stage_bytes + raws) + slab_only;
        c.smem = HDR + 1024 + (size_t)c.stages * stage_bytes + raws + slab_bytes;
    }
    // tensor memory: a second accumulator set if it fits, then more spans of expanded blocks
    const int at = packed ? span * 32 : 0;
    c.nacc = ksplit == 1 && 2 * c.accw + at <= 512 ? 2 : 1;
    c.lag = 1;
    for (int l = 2; packed && l <= 4; l *= 2)
        if (c.stages * c.kps >= l * span && c.nacc * c.accw + l * at <= 512 && l * at <= 256) c.lag = l;
    const int cols = c.nacc * c.accw + c.lag * at;
    if (cols > 512) return c;
    c.tmem_cols = 32;
    while (c.tmem_cols < cols) c.tmem_cols *= 2;
    c.ok = true;
    return c;
}

// Clusters of `size` blocks that can run at a time (one block per SM): the SMs of a cluster lie in one GPC, so fewer than
// sms / size.  Asked of the driver once per device.
int max_clusters(int size, int sms) {
    static std::atomic<int> cached[64][4] = {};   // (any thread; all find the same number)
    int dev = 0;
    const int k = size == 2 ? 1 : size == 4 ? 2 : 3;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sms / (2 * size);
    int n = cached[dev][k].load(std::memory_order_relaxed);
    if (!n) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(size * (sms / size)));
        cfg.blockDim = dim3((unsigned)gemm_threads(FMT_FP16));
        cfg.dynamicSmemBytes = SMEM_LIMIT;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, linear_gemm_tc_kernel<FMT_FP16, false>, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sms / (2 * size);
        }
        cached[dev][k].store(n, std::memory_order_relaxed);
    }
    return n;
}

// What a choice costs, in SM clocks, to compare choices with.  Fitted to timings of tiles between 64 x 896 x 896 and
// 2048 x 151936 x 896: a launch 4000 or 6500; an SM takes in 58 bytes per clock (the two operands of a K block; that, not the tensor
// core, sets the pace of 128 x 256 tiles too); the fp16 issuer needs 360 per K block, the expanding warps 420; a block's
// epilogue 400 and 10 per token; a split tile's exchange 3000 and 14 per token.
double gemm_cost(int fmt, const GemmConfig& c, int row_tiles, int K, int sms) {
    const int nkb = (K + BK - 1) / BK;
    const double blocks = (double)((nkb + c.ksplit - 1) / c.ksplit);
    double per = ((c.duo ? c.bn / 2 : c.bn) * 128.0 + (fmt == FMT_FP16 ? 16384.0 : fmt == FMT_INT8 ? 8192.0 : 4608.0)) / 58.0;
    if (2.0 * c.bn > per) per = 2.0 * c.bn;
    const double least = fmt == FMT_FP16 ? 360.0 : c.lag >= 2 ? 420.0 : 700.0;
    if (per < least) per = least;
    const int tiles = row_tiles * c.ntok;
    const double epi = c.bn / c.fin * 10.0 + 400.0, tile = blocks * per;
    // (a launch of at most half the SMs starts on the ones that the launch before it leaves free)
    const double fixed = tiles * c.ksplit <= sms / 2 ? 4000.0 : 6500.0;
    if (c.ksplit > 1) return tiles > max_clusters(c.ksplit, sms) ? 1e30 : fixed + 3000.0 + 14.0 * c.bn + tile + epi;
    const int at_a_time = c.duo ? max_clusters(2, sms) : sms, waves = ((c.duo ? (row_tiles + 1) / 2 * c.ntok : tiles) + at_a_time - 1) / at_a_time;
    return fixed + (c.nacc == 2 ? waves * (tile > epi ? tile : epi) + epi : waves * (tile + epi));
}

GemmConfig gemm_choose(int fmt, int trows, int M, int row_tiles, int K, int sms) {
    const int units = ((K + BK - 1) / BK + span_blocks(fmt) - 1) / span_blocks(fmt);
    GemmConfig best = {};
    double best_cost = 1e30;
    for (int ks = 1; ks <= 8; ks *= 2) {
        if (ks > 1 && (ks > units || row_tiles * ks > sms)) break;
        int last = 0;
        for (int ntok = (M + 255) / 256; ntok <= (M + 15) / 16; ++ntok) {
            const int bn = ((M + ntok - 1) / ntok + 15) / 16 * 16;
            if (bn == last) continue;
            last = bn;
            // Two blocks on one 256-row tile (cta_group::2): each loads half of the tile's tokens, so a K block of 256 tokens is 32 KB
            // per SM instead of 48 and the tensor core sets the pace instead of the copies: 2048 x 151936 x 896 in fp16 576 -> 500 us,
            // 256 x 151936 x 896 in int8 101 -> 90.  Starting and ending in pairs costs some 3 us (the gate and up of a 512-token
            // prompt, one wave of pairs: 14 -> 17 us), which long calls only, from four waves on, win back.
            const bool long_call = (row_tiles + 1) / 2 * ntok >= 4 * max_clusters(2, sms);
            for (int duo = 0; duo <= (ks == 1 && bn % 32 == 0 && long_call ? 1 : 0); ++duo) {
                const GemmConfig c = gemm_geometry(fmt, trows, M, K, bn, ks, duo != 0);
                if (!c.ok) continue;
                const double cost = gemm_cost(fmt, c, row_tiles, K, sms);
                if (cost < best_cost) {
                    best_cost = cost;
                    best = c;
                }
            }
            if (row_tiles * ntok > 4 * sms && best.ok) break;   // more tiles only re-read the weights
        }
    }
    return best;
}

// The choice for a shape, kept (a choice is a function of its arguments alone): trying all tilings takes the host microseconds,
// and a model asks for the same few shapes over and over.
GemmConfig gemm_config(int fmt, int trows, int M, int row_tiles, int K, int sms) {
    struct Slot {
        int key[6];
        GemmConfig c;
    };
    constexpr int SLOTS = 256;
    static thread_local std::unique_ptr<Slot[]> slots;   // given back when the thread ends
    if (!slots) slots = std::make_unique<Slot[]>(SLOTS);
    const int key[6] = {fmt + 1, trows, M, row_tiles, K, sms};
    uint32_t h = 0;
    for (int v : key) h = (h ^ (uint32_t)v) * 0x9E3779B1u, h ^= h >> 15;
    Slot& s = slots[h % SLOTS];
    if (memcmp(s.key, key, sizeof(key)) != 0) {
        s.c = gemm_choose(fmt, trows, M, row_tiles, K, sms);
        memcpy(s.key, key, sizeof(key));
    }
    return s.c;
}

template <int WFMT, bool DUO>
cudaError_t launch_one(const GemmMaps& mp, const GemmArgs& g, int grid, size_t smem, bool pdl, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)gemm_threads(WFMT));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (DUO || g.ksplit > 1) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = DUO ? 2u : (unsigned)g.ksplit;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&cfg, linear_gemm_tc_kernel<WFMT, DUO>, mp, g);
}

cudaError_t launch_fmt(int fmt, bool duo, const GemmMaps& mp, const GemmArgs& g, int grid, size_t smem, bool pdl, cudaStream_t st) {
    if (fmt == FMT_FP16) return duo ? launch_one<FMT_FP16, true>(mp, g, grid, smem, pdl, st) : launch_one<FMT_FP16, false>(mp, g, grid, smem, pdl, st);
    if (fmt == FMT_INT8) return duo ? launch_one<FMT_INT8, true>(mp, g, grid, smem, pdl, st) : launch_one<FMT_INT8, false>(mp, g, grid, smem, pdl, st);
    return duo ? launch_one<FMT_Q4, true>(mp, g, grid, smem, pdl, st) : launch_one<FMT_Q4, false>(mp, g, grid, smem, pdl, st);
}

}  // namespace

cudaError_t gemm_tc_configure() {
    cudaError_t e = cudaSuccess;
#define CFG(F) \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(linear_gemm_tc_kernel<F, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT); \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(linear_gemm_tc_kernel<F, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
    CFG(FMT_FP16) CFG(FMT_INT8) CFG(FMT_Q4)
#undef CFG
    return e;
}

bool gemm_tc_supported(int fmt, const LinArgs& a, int M) {
    const int K = a.K;
    if (M <= 16 || K < 64 || (K % 8) != 0) return false;
    if (fmt == FMT_INT8 && (K % 16) != 0) return false;   // packed rows keep a 16-byte pitch for the tensor copies
    if (fmt == FMT_Q4 && (K % 32) != 0) return false;
    if (a.norm_w || a.argmax_slot) return false;
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!al16(a.x)) return false;
    for (int i = 0; i < a.nseg; ++i)
        if (a.seg[i].N < 1 || !al16(a.seg[i].W) || !a.seg[i].out) return false;
    return a.epi != EPI_SWIGLU || al16(a.W2);
}

cudaError_t launch_gemm_tc(int fmt, const LinArgs& a, int M, bool overlap, cudaStream_t st) {
    const bool dual = a.epi == EPI_SWIGLU;
    const int K = a.K, sms = current_sm_count();
    if (a.npeer < 0 || a.npeer > 7) return cudaErrorInvalidValue;
    GemmMaps mp;
    GemmArgs g = {};
    // The epilogue goes through a staging tile in shared memory and tensor stores when the output rows keep 16-byte
    // pitch and alignment (lane-by-lane stores otherwise).
    bool aligned = true;
    const int trows = dual ? BM / 2 : BM;   // output columns per tile
    int rows = 0;                           // row tiles
    for (int i = 0; i < a.nseg; ++i) {
        aligned = aligned && (a.seg[i].ld_out % 8) == 0 && (reinterpret_cast<uintptr_t>(a.seg[i].out) & 15) == 0;
        g.seg[i].scale = a.seg[i].scale;
        g.seg[i].bias = a.seg[i].bias;
        g.seg[i].out = a.seg[i].out;
        g.seg[i].N = a.seg[i].N;
        g.seg[i].ld = a.seg[i].ld_out;
        g.seg[i].tile0 = rows;
        rows += (a.seg[i].N + trows - 1) / trows;
    }
    for (int p = 0; p < a.npeer; ++p) {
        aligned = aligned && (reinterpret_cast<uintptr_t>(a.peer_out[p]) & 15) == 0;
        g.peer_out[p] = a.peer_out[p];
    }
    g.scale2 = a.scale2;
    g.nseg = a.nseg;
    g.M = M;
    g.K = K;
    g.rows = trows;
    g.npeer = a.npeer;
    g.sig = a.sig;
    g.epi = a.epi;
    g.status = a.status;
    g.tma_store = aligned ? 1 : 0;
    const GemmConfig c = gemm_config(fmt, trows, M, rows, K, sms);   // the same for a call with peers: the same order of the sums
    if (!c.ok) return cudaErrorInvalidValue;
    g.bn = c.bn;
    g.ntok = c.ntok;
    g.ksplit = c.ksplit;
    g.fin = c.fin;
    g.stages = c.stages;
    g.raw_stages = c.raw_stages;
    g.kps = c.kps;
    g.lag = c.lag;
    g.accw = c.accw;
    g.nacc = c.nacc;
    g.tmem_cols = c.tmem_cols;
    g.slab = c.slab;
    g.two_slabs = c.two_slabs;
    g.swap_off = c.swap_off;
    g.xchg_off = c.xchg_off;
    size_t wbytes = 0;
    for (int i = 0; i < a.nseg; ++i) wbytes += (size_t)a.seg[i].N * (size_t)(fmt == FMT_FP16 ? K * 2 : fmt == FMT_INT8 ? K : K / 2);
    g.evict_first = c.ntok == 1 && wbytes > ((size_t)96 << 20) ? 1 : 0;
    auto weight_map = [&](CUtensorMap* m, const uint8_t* W, int N) {
        if (fmt == FMT_FP16) return encode_tiled_2d(m, true, W, (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, BK, (uint32_t)trows);
        const uint64_t rb = (uint64_t)(fmt == FMT_INT8 ? K : K / 2);
        return encode_tiled_2d(m, false, W, rb, (uint64_t)N, rb, 128, (uint32_t)trows);
    };
    for (int i = 0; i < a.nseg; ++i) {
        if (!weight_map(&mp.w[i], a.seg[i].W, a.seg[i].N)) return cudaErrorInvalidValue;
        if (g.tma_store && !encode_tiled_2d(&mp.out[i], true, a.seg[i].out, (uint64_t)a.seg[i].N, (uint64_t)M, (uint64_t)a.seg[i].ld_out * 2, (uint32_t)trows,
                                            (uint32_t)c.slab, /*swizzle128=*/false))
            return cudaErrorInvalidValue;
    }
    if (dual && !weight_map(&mp.w[1], a.W2, a.seg[0].N)) return cudaErrorInvalidValue;
    const uint16_t* sbase[4];
    int pitch = 0;
    if (fmt == FMT_Q4 && q4_scale_views(a, sbase, &pitch)) {
        g.scale_tma = 1;
        for (int i = 0; i < a.nseg; ++i)
            if (!make_scale_map(&mp.sc[i], sbase[i], a.seg[i].N, pitch, 16, trows)) g.scale_tma = 0;
        if (dual && !make_scale_map(&mp.sc[1], sbase[3], a.seg[0].N, pitch, 16, trows)) g.scale_tma = 0;
    }
    if (!encode_tiled_2d(&mp.x, true, a.x, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, BK, (uint32_t)(c.duo ? c.bn / 2 : c.bn))) return cudaErrorInvalidValue;
    g.tiles = (c.duo ? (rows + 1) / 2 : rows) * c.ntok;
    int grid = g.tiles * c.ksplit;
    const int at_a_time = c.duo ? max_clusters(2, sms) : sms;
    if (c.ksplit == 1 && grid > at_a_time) grid = at_a_time;   // persistent: one block (pair) per SM (pair) walks the tiles
    if (c.duo) grid *= 2;
    return launch_fmt(fmt, c.duo, mp, g, grid, c.smem, overlap, st);
}

}  // namespace nnb
