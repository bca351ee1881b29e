// Wide candidate windows on the tensor cores.
//
// In an open search thousands of spectra share most of their candidates, so
// scoring is a contraction: scores[spectrum][candidate] = sum over bins of
// x[spectrum][bin] * weight[candidate][bin], 2,000-odd bins of which a
// candidate touches some 200.  The list scorer (lists.cu) gathers them from
// shared memory, 16 random bytes per entry and eight spectra, and is bound by
// the shared-memory wavefronts of those gathers (open windows: 2.6e10 pairs/s).
// Here the candidate's list is spread into a dense row of 8-bit weights and 128
// spectra are scored against it by tcgen05.mma (kind::f8f6f4, FP32
// accumulators in tensor memory): 20 times the multiplications, at 300 times
// the rate.
//
// Operands.  The weights 10, 25 and 50 are 5 times 2, 5 and 10, which E4M3
// holds exactly.  A row value x (|x| <= 50.4) is scaled by 8 and split into
// 8-bit pieces, each the rounded remainder of the ones before it, which the MMAs
// add up in one accumulator.  Of a value in [2^e, 2^(e+1)) they leave at most
//   2 pieces (E4M3, E5M2)          2^(e-8),  as BF16 does, from 0.004 on,
//   3 pieces (2 E4M3, E5M2)        2^(e-13), FP16: 2^(e-11), from 0.06 on,
//   6 pieces (3 E4M3, 3 E5M2)      1e-6, for FP32 rows,
// and 8e-6 (1e-6 with six) of smaller ones; over values spread evenly in their
// exponents the RMS error is 0.76 of BF16's and 0.14 of FP16's, and six pieces
// move a score by about 1e-8 of itself (FP32 summation: 6e-8).  The scores only
// choose the candidates that FP32 rescoring orders in the canonical order.
//
// FP32 searches keep 32 candidates for at most 16 results, and the results have
// to be those of scoring every pair in FP32: after the rescoring k_dense_prove
// bounds how far a score of the pieces can be from the FP32 score, and a spectrum
// whose last result is not above the 32nd kept score by more than that (spectra of
// a few peaks, where hundreds of candidates tie) is scored again by the list
// scorer.
//
// Work.  An item is 128 spectra times a run of candidates, taken 512 at a time
// (512 columns of 128 FP32 accumulators fill the SM's tensor memory).  For each
// 128-bin chunk 512 threads, one candidate each, walk their ascending list and
// store the chunk's weights into the operand's 128-byte row (swizzled as
// tcgen05 reads it, so a row's bins spread over all banks), while the MMAs of
// the chunk before run; the spectra's pieces stream from L2 in 16 KB bulk
// copies.  Four more warps read the finished accumulators, lane = spectrum, and
// offer what reaches the spectrum's threshold to its list of the best K.
//
// Measured (20,000 proteins, 80 % +-10 ppm and 20 % +-500 Da windows, all
// scoring): 20,000 spectra in BF16 70.1 -> 13.5 ms, 3,001 in FP32 24.4 -> 13.5 ms.
// A chunk takes about 5,700 cycles, 2,050 of them MMAs (6,100 of FP32's six
// pieces): spreading the lists bounds the rest, its byte stores and list loads
// (3,200 shared-memory cycles), then the epilogue (a quarter).
#include <algorithm>
#include <cuda_fp8.h>

#include "hfx_internal.h"
#include "device_common.cuh"
#include "batched.h"
#include "batched_common.cuh"
#include "lists.h"
#include "lists_device.cuh"
#include "dense.h"

namespace hfx {

constexpr int kDenseRows = 512;                    // candidates per pass
constexpr uint32_t kDenseChunkBytes = kDenseRows * 128;       // one chunk of weights
constexpr uint32_t kPieceBytes = kDenseSpectra * 128;         // one chunk of one piece
constexpr int kPieceStages = 4;
constexpr int kSpreadWarps = kDenseRows / 32;      // warps that spread lists
constexpr int kDenseThreads = (kSpreadWarps + 6) * 32;        // + 4 epilogue, MMA, copies
constexpr int kWindow = 6;                         // list loads (eight entries each) in flight per candidate
constexpr float kDenseScale = 8.0f;                // of the row values (the accumulators hold 8/5 of the scores)

// Offset of byte k of row r within one chunk: 8-row groups of 1,024 bytes, the
// row's eight 16-byte pieces XOR-ed by the row (tcgen05's 128-byte swizzle).
__host__ __device__ __forceinline__ uint32_t swizzled(uint32_t r, uint32_t k) {
    return (r >> 3) * 1024u + (r & 7u) * 128u + (((k >> 4) ^ (r & 7u)) << 4) + (k & 15u);
}

// ---- planning ----

// The dense path pays from some 17 spectra per candidate row on: a row costs
// 0.64 ns whatever the block's windows (18 M rows in 10.5 ms), a pair of the list
// scorer 0.038 ns.  With the line at 16 the +-3 Da blocks of 10,000 spectra that
// passed it made their scoring slower (2.78 -> 3.15 ms); at 32 none of them does,
// and open windows have 36 to 115 (kDenseMinPairs).  A union of fewer than eight
// passes is left to the list scorer too: its pairs with 128 spectra take that
// 20 us, as long as one pass of an SM.
constexpr uint32_t kDenseMinWidth = 4096;

__global__ void k_dense_clear(DenseWs dw, int32_t nspec) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 32ll * nspec) dw.best[i] = 0ull;
    if (i < nspec) {
        dw.kth[i] = 0ull;
        dw.lock[i] = i == 0 && (*dw.hold & 0xFFu) ? 2u : 0u;
    }
    if (i == 0) *dw.n_tiles = *dw.counter = dw.item_off[dw.cap_blocks] = 0u;
}

// One warp per block.  Classes as in k_groups.
__global__ void k_dense_plan(const SpecMeta *__restrict__ meta, const uint32_t *__restrict__ wb,
                             const uint32_t *__restrict__ we, int32_t G, const uint32_t *__restrict__ bucket_end,
                             int32_t nclass, int32_t nbucket, const int32_t *__restrict__ perm,
                             GroupInfo *__restrict__ groups, uint32_t *__restrict__ nchunks, DenseWs dw) {
    const int lane = threadIdx.x & 31;
    const int32_t b = (int32_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    if (b >= dw.cap_blocks) return;
    if (lane == 0) dw.item_off[b] = 0u;
    // the class of block b, its first spectrum and first group
    uint32_t nb = 0, ng = 0, start = 0, mine = ~0u, pos0 = 0, cnt = 0, g0 = 0;
    for (int c = 0; c < nclass; ++c) {
        const uint32_t end = bucket_end[(c + 1) * nbucket - 1];
        const uint32_t n = end - start, blocks = (n + kDenseSpectra - 1) / kDenseSpectra;
        if (mine == ~0u && (uint32_t)b < nb + blocks) {
            mine = (uint32_t)b - nb;
            pos0 = start + mine * kDenseSpectra;
            cnt = min((uint32_t)kDenseSpectra, end - pos0);
            g0 = ng + mine * (kDenseSpectra / (uint32_t)G);
        }
        nb += blocks;
        ng += (n + (uint32_t)G - 1) / (uint32_t)G;
        start = end;
    }
    if (mine == ~0u) return;
    uint32_t lo = ~0u, hi = 0u;
    unsigned long long pairs = 0;
    int32_t maxlen = 0, odd = 0, charges = 0;
    for (uint32_t j = lane; j < cnt; j += 32) {
        const int32_t s = perm[pos0 + j];
        const uint32_t a = wb[s], e = we[s];
        if (e > a) {
            lo = min(lo, a);
            hi = max(hi, e);
            pairs += e - a;
        }
        maxlen = max(maxlen, meta[s].len);
        odd |= meta[s].nonfinite;
        charges = meta[s].charges_plain;
    }
    lo = __reduce_min_sync(kFullMask, lo);
    hi = __reduce_max_sync(kFullMask, hi);
    maxlen = __reduce_max_sync(kFullMask, maxlen);
    odd = __reduce_or_sync(kFullMask, (uint32_t)odd);
    charges = __reduce_max_sync(kFullMask, charges);
    for (int o = 16; o >= 1; o >>= 1) pairs += __shfl_xor_sync(kFullMask, pairs, o);
    // a NaN of one row would reach every candidate's score (0 x NaN)
    if (hi <= lo || hi - lo < kDenseMinWidth || charges < 1 || odd ||
        pairs < (unsigned long long)kDenseMinPairs * (hi - lo))
        return;
    for (uint32_t g = lane; g < (cnt + (uint32_t)G - 1) / (uint32_t)G; g += 32) {
        groups[g0 + g].block = b;
        nchunks[g0 + g] = 0u;
    }
    if (lane == 0) {
        DenseBlock d;
        d.pos0 = pos0;
        d.count = cnt;
        d.lo = lo;
        d.hi = hi;
        d.maxlen = maxlen;
        d.charges = charges;
        // items of about the same cost: passes x chunks of a row near 136, less
        // when that leaves fewer than twelve items for each SM
        const unsigned long long share = (unsigned long long)(hi - lo) * nb / (12u * 152u) / kDenseRows;
        const uint32_t even = 136u / (((uint32_t)maxlen + 127u) / 128u);
        d.chunk = max((uint32_t)min(share, (unsigned long long)even), 1u) * kDenseRows;
        d.tile = atomicAdd(dw.n_tiles, 1u);
        d.ladder = 0u;
        dw.blocks[b] = d;
        dw.tile_block[d.tile] = (uint32_t)b;
        dw.item_off[b] = (hi - lo + d.chunk - 1) / d.chunk;
    }
}

// ---- operand tiles: [tile][chunk][piece], swizzled as above ----

// Pieces in E4M3; the others, finer ones in E5M2.
constexpr int dense_e4m3(int P) { return P / 2 + (P == 3 ? 1 : 0); }

template <int P>
__global__ void __launch_bounds__(256) k_dense_pack(const float *__restrict__ rows, int64_t stride,
                                                    const int32_t *__restrict__ perm, DenseWs dw, uint32_t cap_tiles,
                                                    uint8_t *__restrict__ tiles, uint32_t *__restrict__ err) {
    const uint32_t t = blockIdx.x, chunk = blockIdx.y;
    const uint32_t n = *dw.n_tiles;
    if (t == 0 && chunk == 0 && threadIdx.x == 0 && n > cap_tiles) atomicOr(err, kErrBounds);
    if (t >= n) return;
    const DenseBlock d = dw.blocks[dw.tile_block[t]];
    uint8_t *out = tiles + ((size_t)t * gridDim.y + chunk) * P * kPieceBytes;
    for (uint32_t u = threadIdx.x; u < kDenseSpectra * 8u; u += blockDim.x) {
        const uint32_t r = u >> 3, q = u & 7u;
        float x[16];
        const int64_t bin = (int64_t)chunk * 128 + q * 16;
        if (r < d.count && bin < stride) {
            const float4 *src = reinterpret_cast<const float4 *>(rows + (size_t)perm[d.pos0 + r] * stride + bin);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = src[i];
                x[4 * i] = v.x;
                x[4 * i + 1] = v.y;
                x[4 * i + 2] = v.z;
                x[4 * i + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __fmul_rn(x[i], kDenseScale);
#pragma unroll
        for (int p = 0; p < P; ++p) {
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                constexpr __nv_fp8_interpretation_t kinds[2] = {__NV_E4M3, __NV_E5M2};
                const __nv_fp8_interpretation_t kind = kinds[p < dense_e4m3(P) ? 0 : 1];
                const __nv_fp8_storage_t c = __nv_cvt_float_to_fp8(x[i], __NV_SATFINITE, kind);
                x[i] = __fsub_rn(x[i], __half2float(__half(__nv_cvt_fp8_to_halfraw(c, kind))));
                w[i >> 2] |= (uint32_t)c << (8 * (i & 3));
            }
            *reinterpret_cast<uint4 *>(out + (size_t)p * kPieceBytes + swizzled(r, q * 16)) =
                make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// ---- tcgen05 ----

__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    // start address, stride of 1,024 bytes between 8-row groups, 128-byte swizzle
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// D = F32, A (spectra) = E4M3 or E5M2, B (candidates) = E4M3, both K-major, M = 128, N = 256.
constexpr uint32_t kDenseE5M2 = 1u << 7;
constexpr uint32_t kDenseIdesc = (1u << 4) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_f8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_load32(uint32_t addr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float tmem_load1(uint32_t addr) {
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r)
                 : "r"(addr)
                 : "memory");
    return __uint_as_float(r);
}
__device__ __forceinline__ float max_nan(float a, float b, float c) {
    float m;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}
// A candidate as one key: the larger is the better (score, then the smaller
// position); 0: none.
__device__ __forceinline__ unsigned long long packed(float score, uint32_t p) {
    return (unsigned long long)score_order(score) << 32 | (uint32_t)~p;
}
__device__ __forceinline__ float score_of(uint32_t order) {  // inverse of score_order, 0 = none yet
    if (order == 0u) return -INFINITY;
    return __uint_as_float((order & 0x80000000u) ? (order & 0x7FFFFFFFu) : ~order);
}

// Barriers of the pipeline (shared memory).
struct DenseBars {
    uint64_t piece_full[kPieceStages], piece_empty[kPieceStages];  // the spectra's pieces
    uint64_t rows_full[2], rows_empty[2];                          // the candidates' weights
    uint64_t acc_full, acc_empty;                                  // the accumulators
    uint64_t drain;                                                // MMAs in flight when a wait gave up
};

constexpr uint32_t kDenseWaitLimit = 1u << 21;
// Waits for a phase: false after kDenseWaitLimit polls, or when another wait of
// the CTA has given up.
__device__ __forceinline__ bool dense_wait(uint64_t *bar, uint32_t phase, volatile uint32_t *give_up, uint32_t *err) {
    for (uint32_t i = 0; i < kDenseWaitLimit; ++i) {
        if (mbar_wait(bar, phase, 1u)) return true;
        if ((i & 63u) == 63u && *give_up) return false;
    }
    *give_up = 1u;
    atomicOr(err, kErrTimeout);
    return false;
}
// The same for a whole warp: every lane polls, and so sees what the phase
// publishes, and all lanes go on or all give up -- the warp-wide steps that
// follow need every lane.
__device__ __forceinline__ bool dense_wait_warp(uint64_t *bar, uint32_t phase, volatile uint32_t *give_up,
                                                uint32_t *err) {
    for (uint32_t i = 0; i < kDenseWaitLimit; ++i) {
        if (__all_sync(kFullMask, mbar_wait(bar, phase, 1u))) return true;
        if ((i & 63u) == 63u && __any_sync(kFullMask, *give_up != 0u)) return false;
    }
    if ((threadIdx.x & 31) == 0) {
        *give_up = 1u;
        atomicOr(err, kErrTimeout);
    }
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Shared memory after the barriers' 1,024 bytes: two chunks of weights, the
// piece stages, and a queue per spectrum.
constexpr size_t kDenseSmem = 1024 + 2 * (size_t)kDenseChunkBytes + kPieceStages * (size_t)kPieceBytes +
                              kDenseSpectra * kDenseQueue * (size_t)8;

template <int P>
__global__ void __launch_bounds__(kDenseThreads, 1)
k_dense_score(const uint16_t *__restrict__ lists, uint64_t list_total, const uint32_t *__restrict__ lstart,
              uint64_t total10, const uint16_t *__restrict__ list_len, uint32_t num_pep,
              const uint8_t *__restrict__ tiles, uint32_t cap_tiles, uint32_t tile_chunks,
              const uint32_t *__restrict__ wb, const uint32_t *__restrict__ we, const int32_t *__restrict__ perm,
              DenseWs dw, int32_t K, unsigned long long *__restrict__ stats, uint32_t *__restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    DenseBars &bar = *reinterpret_cast<DenseBars *>(smem);
    uint8_t *rows = smem + 1024, *pieces = rows + 2 * kDenseChunkBytes;
    unsigned long long *q = reinterpret_cast<unsigned long long *>(pieces + kPieceStages * kPieceBytes);  // [128][kDenseQueue]
    __shared__ uint32_t s_item, s_tmem;
    __shared__ volatile uint32_t s_give_up;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kPieceStages; ++i) {
            mbar_init(&bar.piece_full[i], 1);
            mbar_init(&bar.piece_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar.rows_full[i], kSpreadWarps);
            mbar_init(&bar.rows_empty[i], 1);
        }
        mbar_init(&bar.acc_full, 1);
        mbar_init(&bar.acc_empty, 4);
        mbar_init(&bar.drain, 1);
        s_give_up = 0u;
    }
    if (warp == kSpreadWarps + 4) {  // the MMA warp owns the tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t total = dw.item_off[dw.cap_blocks];
    // Items are taken in an order that hops between the blocks: in their own
    // order all CTAs would start on one block's 128 spectra at once, without a
    // threshold and waiting for each other's locks (15.9 against 10.5 ms for the
    // open windows of 20,000 spectra).
    uint32_t hop = max(1u, (uint32_t)((unsigned long long)total * 618 / 1000));
    for (uint32_t x = hop, y = total; y != 0u || x != 1u;) {  // a step without a common divisor
        if (y == 0u) {
            ++hop;
            x = hop;
            y = total;
        }
        const uint32_t r = y ? x % y : 0u;
        x = y ? y : x;
        y = r;
        if (total <= 1u) break;
    }
    // each role counts the chunks, pieces and passes it has handled; the
    // counts give the buffer and the barrier phase
    uint32_t n_chunk = 0, n_piece = 0, n_pass = 0;
    unsigned long long my_rows = 0, my_entries = 0, my_pairs = 0;
    // epilogue warps: the item's spectrum of this lane, its window, the key that
    // a candidate has to exceed (its list's K-th) and its queue.  Spectra of a few
    // peaks have thousands of candidates tied with the K-th: those behind it are
    // not looked at (cut), or the merging of them would take ten times the rest
    const uint32_t m = threadIdx.x & (kDenseSpectra - 1u);
    int32_t s = -1;
    uint32_t a = 0, e = 0, qn = 0;
    unsigned long long floor_key = ~0ull;
    // the least score that is kept at positions from p on
    auto cut_from = [&](uint32_t p) {
        const uint32_t order = (uint32_t)(floor_key >> 32);
        if (order == ~0u) return INFINITY;
        return score_of(order + (order != 0u && (uint32_t)~(uint32_t)floor_key < p ? 1u : 0u));
    };
    // Merges lane j's queue into its spectrum's list (warp-wide).
    auto merge = [&](int j) {
        const int cnt = (int)__shfl_sync(kFullMask, qn, j);
        const int32_t sj = __shfl_sync(kFullMask, s, j);
        unsigned long long x = lane < cnt ? q[((m & ~31u) + (uint32_t)j) * kDenseQueue + lane] : 0ull;
        // the queue, best first in lanes 0 .. 15
#pragma unroll
        for (int w = 2; w <= kDenseQueue; w <<= 1)
#pragma unroll
            for (int o = w >> 1; o > 0; o >>= 1) {
                const unsigned long long y = __shfl_xor_sync(kFullMask, x, o);
                const bool high = ((lane & o) == 0) == ((lane & w) == 0);
                x = high ? max(x, y) : min(x, y);
            }
        uint32_t got = 0u;
        if (lane == 0)
            for (uint32_t i = 0; i < kLockLimit && !got; ++i) {
                got = atomicCAS(dw.lock + sj, 0u, 1u) == 0u;
                // the search has failed already: the other locks need not run out too
                if ((i & 255u) == 255u && (*(volatile uint32_t *)err & kErrTimeout)) break;
            }
        got = __shfl_sync(kFullMask, got, 0);
        if (!got) {
            if (lane == 0) atomicOr(err, kErrTimeout);
            if (lane == j) qn = 0;
            return;
        }
        __threadfence();
        unsigned long long *list = dw.best + (size_t)sj * 32;
        unsigned long long l = __ldcg(list + lane);
        l = max(l, __shfl_sync(kFullMask, x, 31 - lane));  // the best 32 of both, bitonic
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(kFullMask, l, o);
            l = (lane & o) == 0 ? max(l, y) : min(l, y);
        }
        __stcg(list + lane, l);
        const unsigned long long kth = __shfl_sync(kFullMask, l, K - 1);
        if (lane == 0) __stcg(dw.kth + sj, kth);
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(dw.lock + sj, 0u);
        if (lane == j) {
            qn = 0;
            floor_key = max(floor_key, kth);
        }
        __syncwarp();
    };
    while (true) {
        if (threadIdx.x == 0) s_item = atomicAdd(dw.counter, 1u);
        if (__syncthreads_or((int)s_give_up)) break;
        if (s_item >= total) break;
        const uint32_t item = (uint32_t)((unsigned long long)s_item * hop % total);
        const int32_t b = find_group(dw.item_off, dw.cap_blocks, item);
        const DenseBlock d = dw.blocks[b];
        const uint32_t p0 = d.lo + (item - dw.item_off[b]) * d.chunk;
        const uint32_t p1 = min(d.hi, p0 + d.chunk);
        const uint32_t chunks = d.tile < cap_tiles ? (uint32_t)(d.maxlen + 127) / 128u : 0u;  // none: reported by the packing
        const uint32_t passes = chunks ? (p1 - p0 + kDenseRows - 1) / kDenseRows : 0u;
        if (warp < kSpreadWarps) {
            // ---- lists -> weights: thread = candidate ----
            const uint32_t t = threadIdx.x;
            const uint32_t row0 = smem_u32(rows) + (t >> 3) * 1024u + (t & 7u) * 128u, sw = t & 7u;
            const uint16_t *llen = list_len + (size_t)(d.charges - 1) * num_pep;
            for (uint32_t pass = 0; pass < passes; ++pass) {
                const uint32_t p = p0 + pass * kDenseRows + t;
                uint32_t n = 0;
                const uint16_t *lp = lists;
                if (p < p1 && p < num_pep) {
                    n = llen[p];
                    const uint64_t off = list_offset(lstart, total10, d.charges, p);
                    if (off + n > list_total) {
                        atomicOr(err, kErrBounds);
                        n = 0;
                    } else {
                        lp += off;
                    }
                    my_rows += 1;
                    my_entries += n;
                }
                // A window of 48 entries in registers (six loads).  After a chunk
                // the loads it has used up are replaced behind the others, so a
                // load's latency lies behind the next chunk and nothing is read
                // twice.  (One load at a time, or the whole window anew per
                // chunk, left the warps waiting for list loads.)  Past the end:
                // a bin no chunk holds.
                uint32_t at = 0;
                uint4 v[kWindow];
                auto load8 = [&](uint32_t i) {
                    return i < n ? __ldg(reinterpret_cast<const uint4 *>(lp + i)) : make_uint4(~0u, ~0u, ~0u, ~0u);
                };
                auto pad = [&](uint4 &x, uint32_t i) {
                    const int left = (int)n - (int)i;
                    if (left < 8) {
                        x.x = left < 1 ? ~0u : (left < 2 ? x.x | 0xFFFF0000u : x.x);
                        x.y = left < 3 ? ~0u : (left < 4 ? x.y | 0xFFFF0000u : x.y);
                        x.z = left < 5 ? ~0u : (left < 6 ? x.z | 0xFFFF0000u : x.z);
                        x.w = left < 7 ? ~0u : x.w | 0xFFFF0000u;
                    }
                };
#pragma unroll
                for (int i = 0; i < kWindow; ++i) v[i] = load8(8u * i);
                for (uint32_t c = 0; c < chunks; ++c, ++n_chunk) {
                    const uint32_t buf = n_chunk & 1u;
                    if (!dense_wait_warp(&bar.rows_empty[buf], ((n_chunk >> 1) & 1u) ^ 1u, &s_give_up, err)) goto done;
                    const uint32_t row = row0 + buf * kDenseChunkBytes;
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) sts_u128(row + ((j ^ sw) << 4), make_uint4(0u, 0u, 0u, 0u));
                    // the chunk's entries of eight: 2, 5, 10 in E4M3 for levels 1, 2, 3
                    auto spread = [&](const uint4 &x) {
                        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t e = j & 1 ? w[j >> 1] >> 16 : w[j >> 1] & 0xFFFFu;
                            const uint32_t code = __byte_perm(0x524A4000u, 0u, e & 3u);
                            asm volatile(
                                "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, %3;\n\t@p st.shared.u8 [%0], %1;\n\t}" ::"r"(
                                    row + (((e >> 2) & 127u) ^ (sw << 4))),
                                "r"(code), "r"(e >> 9), "r"(c)
                                : "memory");
                        }
                    };
                    bool more;
                    do {  // again where a chunk holds more than the window
                        if (__any_sync(kFullMask, at + 8u * kWindow > n)) {
#pragma unroll
                            for (int i = 0; i < kWindow; ++i) pad(v[i], at + 8u * i);
                        }
                        // a later load is looked at when some lane used up the
                        // one before it: the last may still be on its way
                        uint32_t used = 0;
#pragma unroll
                        for (uint32_t i = 0; i < kWindow; ++i) {
                            if (i > 0 && !__any_sync(kFullMask, used == i)) break;
                            spread(v[i]);
                            used += used == i && v[i].w >> 25 <= c ? 1u : 0u;
                        }
                        at += 8u * used;
                        more = __any_sync(kFullMask, used == (uint32_t)kWindow);
                        if (__any_sync(kFullMask, used != 0u)) {
#pragma unroll
                            for (uint32_t step = 1; step < kWindow; step <<= 1)
                                if (used & step) {
#pragma unroll
                                    for (uint32_t i = 0; i + step < kWindow; ++i) v[i] = v[i + step];
                                }
#pragma unroll
                            for (uint32_t i = 0; i < kWindow; ++i)
                                if (i + used >= kWindow) v[i] = load8(at + 8u * i);
                        }
                    } while (more);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar.rows_full[buf]);
                }
            }
        } else if (warp < kSpreadWarps + 4) {
            // ---- accumulators -> the best K: lane = spectrum ----
            // Full queues are merged into the spectrum's list in global memory
            // (sorted, under a lock), whose K-th is the threshold of every
            // CTA.  (A list per item started anew every 8,192 candidates:
            // 100,000 cycles of merging a pass.)
            {
                s = m < d.count ? perm[d.pos0 + m] : -1;
                a = s >= 0 ? wb[s] : 0u;
                e = s >= 0 ? we[s] : 0u;
                floor_key = s >= 0 ? 0ull : ~0ull;
                qn = 0;
            }
            for (uint32_t pass = 0; pass < passes; ++pass, ++n_pass) {
                if (s >= 0) floor_key = max(floor_key, __ldcg(dw.kth + s));
                if (!dense_wait_warp(&bar.acc_full, n_pass & 1u, &s_give_up, err)) goto done;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t pb = p0 + pass * kDenseRows;
                const uint32_t pe = min(p1, pb + kDenseRows);
                const uint32_t c0 = max(a, pb) - pb, c1 = max(min(e, pe), pb) - pb;  // this spectrum's columns
                if (c1 > c0) my_pairs += c1 - c0;
                const uint32_t acc = tmem + ((m >> 5) << 21);
                // no threshold yet: the largest of nine cuts between the lowest
                // and the highest score that at least K of this pass reach
                const bool fresh = floor_key == 0ull && c1 >= c0 + (uint32_t)K;
                if (__any_sync(kFullMask, fresh)) {
                    float low = INFINITY, high = -INFINITY;
                    float v[32];
#pragma unroll 1
                    for (uint32_t j0 = 0; j0 < kDenseRows; j0 += 32) {
                        tmem_load32(acc + j0, v);
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (j0 + j >= c0 && j0 + j < c1) {
                                low = fminf(low, v[j]);
                                high = fmaxf(high, v[j]);
                            }
                    }
#pragma unroll 1
                    for (int it = 0; it < 9; ++it) {
                        const float cut = 0.5f * low + 0.5f * high;
                        uint32_t n = 0;
#pragma unroll 1
                        for (uint32_t j0 = 0; j0 < kDenseRows; j0 += 32) {
                            tmem_load32(acc + j0, v);
#pragma unroll
                            for (int j = 0; j < 32; ++j) n += j0 + j >= c0 && j0 + j < c1 && v[j] >= cut ? 1u : 0u;
                        }
                        if (n >= (uint32_t)K) low = cut;
                        else high = cut;
                    }
                    if (fresh) floor_key = (unsigned long long)score_order(low) << 32;
                }
                float cut = cut_from(pb);
#pragma unroll 1
                for (uint32_t j0 = 0; j0 < kDenseRows; j0 += 32) {
                    float v[32];
                    tmem_load32(acc + j0, v);
                    float top = max_nan(v[30], v[31], v[0]);
#pragma unroll
                    for (int j = 1; j < 30; j += 2) top = max_nan(top, v[j], v[j + 1]);
                    // this spectrum's columns of these 32
                    const uint32_t from = c0 > j0 ? min(c0 - j0, 32u) : 0u, to = c1 > j0 ? min(c1 - j0, 32u) : 0u;
                    if (!__any_sync(kFullMask, to > from && !(top < cut))) continue;
                    uint32_t hit = 0;
#pragma unroll
                    for (int j = 0; j < 32; ++j) hit |= v[j] < cut ? 0u : 1u << j;
                    hit &= to > from ? (0xFFFFFFFFu >> (32u - (to - from))) << from : 0u;
                    // the columns some lane keeps, one at a time (read again: a
                    // register is not indexed by a column)
                    for (uint32_t any = __reduce_or_sync(kFullMask, hit); any; any &= any - 1u) {
                        const uint32_t j = (uint32_t)__ffs(any) - 1u;
                        const unsigned long long x = packed(tmem_load1(acc + j0 + j), pb + j0 + j);
                        if (((hit >> j) & 1u) && x > floor_key) q[m * kDenseQueue + qn++] = x;
                        uint32_t full = __ballot_sync(kFullMask, qn == (uint32_t)kDenseQueue);
                        __syncwarp();
                        if (full) {
                            for (; full; full &= full - 1u) merge(__ffs(full) - 1);
                            cut = cut_from(pb);
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar.acc_empty);
            }
            // what is left in the queue goes to the item's own place, for the
            // last merge (under the lock it held up the next accumulators)
            unsigned long long *left = dw.left + ((size_t)item * kDenseSpectra + m) * kDenseQueue;
            for (uint32_t i = 0; i < (uint32_t)kDenseQueue; ++i) left[i] = i < qn ? q[m * kDenseQueue + i] : 0ull;
        } else if (warp == kSpreadWarps + 4) {
            // ---- MMAs ----
            if (lane == 0) {
                for (uint32_t pass = 0; pass < passes; ++pass, ++n_pass) {
                    if (!dense_wait(&bar.acc_empty, (n_pass & 1u) ^ 1u, &s_give_up, err)) goto done;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (uint32_t c = 0; c < chunks; ++c, ++n_chunk) {
                        const uint32_t buf = n_chunk & 1u;
                        if (!dense_wait(&bar.rows_full[buf], (n_chunk >> 1) & 1u, &s_give_up, err)) goto done;
                        const uint32_t rb = smem_u32(rows) + buf * kDenseChunkBytes;
                        for (int p = 0; p < P; ++p, ++n_piece) {
                            const uint32_t st = n_piece % kPieceStages;
                            if (!dense_wait(&bar.piece_full[st], (n_piece / kPieceStages) & 1u, &s_give_up, err)) goto done;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const uint32_t pa = smem_u32(pieces) + st * kPieceBytes;
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k)
#pragma unroll
                                for (uint32_t h = 0; h < 2; ++h)
                                    mma_f8(tmem + h * 256u, operand_desc(pa + 32u * k),
                                           operand_desc(rb + h * (kDenseChunkBytes / 2) + 32u * k),
                                           kDenseIdesc | (p < dense_e4m3(P) ? 0u : kDenseE5M2),
                                           c > 0 || p > 0 || k > 0);
                            mma_commit(smem_u32(&bar.piece_empty[st]));
                        }
                        mma_commit(smem_u32(&bar.rows_empty[buf]));
                    }
                    mma_commit(smem_u32(&bar.acc_full));
                }
            }
        } else if (lane == 0) {
            // ---- the spectra's pieces, L2 -> shared memory ----
            const uint8_t *src = tiles + (size_t)d.tile * tile_chunks * P * kPieceBytes;
            for (uint32_t pass = 0; pass < passes; ++pass)
                for (uint32_t i = 0; i < chunks * P; ++i, ++n_piece) {
                    const uint32_t st = n_piece % kPieceStages;
                    if (!dense_wait(&bar.piece_empty[st], ((n_piece / kPieceStages) & 1u) ^ 1u, &s_give_up, err)) goto done;
                    mbar_arrive_expect_tx(&bar.piece_full[st], kPieceBytes);
                    bulk_g2s(pieces + st * kPieceBytes, src + (size_t)i * kPieceBytes, kPieceBytes, &bar.piece_full[st]);
                }
        }
    done:
        __syncwarp();
        __syncthreads();
    }
    __syncthreads();
    if (s_give_up) {
        // a wait gave up: let copies and MMAs in flight end before the CTA does
        if (warp == kSpreadWarps + 5 && lane == 0)
            for (uint32_t i = n_piece > kPieceStages ? n_piece - kPieceStages : 0u; i < n_piece; ++i)
                mbar_wait(&bar.piece_full[i % kPieceStages], (i / kPieceStages) & 1u, kDenseWaitLimit);
        if (warp == kSpreadWarps + 4 && lane == 0) {
            mma_commit(smem_u32(&bar.drain));
            mbar_wait(&bar.drain, 0u, kDenseWaitLimit);
        }
        __syncwarp();
    }
    __syncthreads();
    if (warp == kSpreadWarps + 4)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    if (stats) {
        for (int o = 16; o >= 1; o >>= 1) {
            my_rows += __shfl_xor_sync(kFullMask, my_rows, o);
            my_entries += __shfl_xor_sync(kFullMask, my_entries, o);
            my_pairs += __shfl_xor_sync(kFullMask, my_pairs, o);
        }
        if (lane == 0) {
            atomicAdd(&stats[2], my_rows);
            atomicAdd(&stats[3], my_entries);
            atomicAdd(&stats[4], my_pairs);
            atomicAdd(&stats[5], my_rows);
            if (warp == kSpreadWarps + 5) atomicAdd(&stats[7], (unsigned long long)n_piece * kPieceBytes);
        }
    }
}

// ---- FP32 searches: are the results certain? ----
//
// A candidate that was not kept has a score of the pieces p of at most p32, the
// 32nd kept one's, and its FP32 score is at most p + E.  With a list of n entries
// and total weight T, N the sum of weight x |x| over the list's negative values and
// M = p32 + N (no partial sum of either is larger):
//   products and accumulators: at most 6 n products that are not zero and one
//     accumulator per MMA, each off by no more than 2^-22 M -- twice the unit of an
//     FP32 sum that truncates (measured: 1.5e-7 of a score, some 10^-4 of E),
//   row values: T 2^-20 (six pieces),
//   the canonical FP32 sum: (n / 32 + 6) 2^-24 (M + N).
// n and T come of the block's longest ladder, L prefixes: 10 L z entries (or all
// bins) and weights 240 L z; N is at most T times the row's lowest value and 50
// times the sum of its negative ones.  Of spectra
// with 50 to 400 peaks (20,000 proteins, +-500 Da) the tenth result lies 570 to
// 2,900 above the 32nd, E is 10 to 200.  The rescored candidates are checked
// against E themselves.  A warp per spectrum, bound by reading its row once.
__global__ void __launch_bounds__(256) k_dense_ladders(const uint32_t *__restrict__ tc, const uint32_t *__restrict__ tn,
                                                       DenseWs dw) {
    const uint32_t b = blockIdx.x;
    if (dw.item_off[b] == dw.item_off[b + 1]) return;  // not dense
    const uint32_t hi = dw.blocks[b].hi;
    uint32_t ladder = 0;
    for (uint32_t p = dw.blocks[b].lo + blockIdx.y * blockDim.x + threadIdx.x; p < hi; p += gridDim.y * blockDim.x)
        ladder = max(ladder, tn[p] > tc[p] ? tn[p] - tc[p] : 0u);
    ladder = __reduce_max_sync(kFullMask, ladder);
    if ((threadIdx.x & 31) == 0) atomicMax(&dw.blocks[b].ladder, ladder);
}

__global__ void __launch_bounds__(128) k_dense_prove(
    const SpecMeta *__restrict__ meta, const int32_t *__restrict__ group_of, const GroupInfo *__restrict__ groups,
    const DenseBlock *__restrict__ blocks, const uint32_t *__restrict__ wb, const uint32_t *__restrict__ we,
    const float *__restrict__ rows, int64_t stride, const float *__restrict__ kept_s, const uint64_t *__restrict__ kept_k, int32_t nspec,
    int32_t topn, const float *__restrict__ out_s, const uint64_t *__restrict__ out_k,
    SpecMeta *__restrict__ open_meta, uint32_t *__restrict__ n_open) {
    constexpr int kKept = 32;
    const int lane = threadIdx.x & 31;
    const int32_t s = (int32_t)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (s >= nspec) return;
    SpecMeta m = meta[s];
    int32_t b = -1;
    if (m.status == 0) b = groups[group_of[s]].block;
    bool certain = true;  // no row, list-scored, or every candidate kept
    if (b >= 0 && we[s] - wb[s] > (uint32_t)kKept) {
        const DenseBlock d = blocks[b];
        float low = 0.0f;
        double neg = 0.0;
        for (int32_t i = lane; i < m.len; i += 32) {
            const float x = fminf(rows[(size_t)s * stride + i], 0.0f);
            low = fminf(low, x);
            neg -= (double)x;
        }
        for (int o = 16; o >= 1; o >>= 1) {
            low = fminf(low, __shfl_xor_sync(kFullMask, low, o));
            neg += __shfl_xor_sync(kFullMask, neg, o);
        }
        const double ions = (double)d.ladder * (double)m.charges_plain, weight = 240.0 * ions;
        const double n = fmin(10.0 * ions, (double)m.len);
        const double to_score = 5.0 / (double)kDenseScale;
        const double p32 = to_score * (double)kept_s[(size_t)s * kKept + kKept - 1];
        const double N = fmin(weight * -(double)low, 50.0 * neg), M = fmax(p32, 0.0) + N;
        const double mmas = 6.0 * 4.0 * (double)((d.maxlen + 127) / 128);
        const double E = 1.01 * ((6.0 * n + mmas) * 0x1p-22 * M + weight * 0x1p-20 +
                                 (n / 32.0 + 6.0) * 0x1p-24 * (M + N));
        certain = (double)out_s[(size_t)s * topn + topn - 1] > p32 + E;
        if (lane < topn) {  // each result's own two scores
            const uint64_t k = out_k[(size_t)s * topn + lane];
            const double f = (double)out_s[(size_t)s * topn + lane];
            bool near = false;
            for (int t = 0; t < kKept; ++t)
                if (kept_k[(size_t)s * kKept + t] == k)
                    near = fabs(to_score * (double)kept_s[(size_t)s * kKept + t] - f) <= E;
            certain = certain && near;
        }
        certain = __all_sync(kFullMask, certain);
    }
    if (lane == 0) {
        if (certain) m.status = -1;
        else atomicAdd(n_open, 1u);
        open_meta[s] = m;
    }
}

__global__ void k_dense_close(const SpecMeta *__restrict__ open_meta, const float *__restrict__ in_s,
                              const uint64_t *__restrict__ in_k, int32_t nspec, int32_t topn,
                              const uint32_t *__restrict__ idx_sorted, float *__restrict__ out_s,
                              uint64_t *__restrict__ out_k, uint32_t *__restrict__ out_pep) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)nspec * topn || open_meta[i / topn].status != 0) return;
    out_s[i] = in_s[i];
    out_k[i] = in_k[i];
    out_pep[i] = in_k[i] != ~0ull ? idx_sorted[in_k[i]] : ~0u;
}

}  // namespace hfx

using namespace hfx;

int hfx_dense_pieces(int elem_kind) { return elem_kind == 1 ? 2 : (elem_kind == 2 ? 3 : 6); }

int hfx_dense_plan(const SpecMeta *meta, int32_t nspec, const uint32_t *wb, const uint32_t *we, int32_t G,
                   const uint32_t *bucket_end, const BatchedWs &ws, uint32_t *nchunks, const DenseWs &dw,
                   cudaStream_t st) {
    const int nclass = 12;
    k_dense_clear<<<(unsigned)((32ll * nspec + 255) / 256), 256, 0, st>>>(dw, nspec);
    k_dense_plan<<<(dw.cap_blocks + 3) / 4, 128, 0, st>>>(meta, wb, we, G, bucket_end, nclass, kBucketCount / nclass,
                                                          ws.perm, ws.groups, nchunks, dw);
    return (int)cudaGetLastError();
}

int hfx_dense_pack(const float *rows, int64_t stride, const BatchedWs &ws, const DenseWs &dw, uint32_t cap_tiles,
                   int pieces, uint8_t *tiles, uint32_t *err, cudaStream_t st) {
    if (cap_tiles == 0) return 0;
    const dim3 grid(cap_tiles, (unsigned)dense_chunks(stride));
    if (pieces == 2) k_dense_pack<2><<<grid, 256, 0, st>>>(rows, stride, ws.perm, dw, cap_tiles, tiles, err);
    else if (pieces == 3) k_dense_pack<3><<<grid, 256, 0, st>>>(rows, stride, ws.perm, dw, cap_tiles, tiles, err);
    else if (pieces == 6) k_dense_pack<6><<<grid, 256, 0, st>>>(rows, stride, ws.perm, dw, cap_tiles, tiles, err);
    else return (int)cudaErrorInvalidValue;
    return (int)cudaGetLastError();
}

int hfx_dense_score(const uint16_t *lists, uint64_t list_total, const uint32_t *lstart, uint64_t total10,
                    const uint16_t *list_len, uint32_t num_pep, const uint8_t *tiles, uint32_t cap_tiles,
                    int64_t stride, int pieces, const uint32_t *wb, const uint32_t *we, const BatchedWs &ws,
                    const DenseWs &dw, int32_t K, unsigned long long *stats, uint32_t *err, cudaStream_t st) {
    if (cap_tiles == 0) return 0;
    if (K > 32) return (int)cudaErrorInvalidValue;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto f = pieces == 2 ? k_dense_score<2> : (pieces == 3 ? k_dense_score<3> : k_dense_score<6>);
    const size_t smem = kDenseSmem + 1024;
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    f<<<sms, kDenseThreads, smem, st>>>(lists, list_total, lstart, total10, list_len, num_pep, tiles, cap_tiles,
                                        (uint32_t)dense_chunks(stride), wb, we, ws.perm, dw, K, stats, err);
    return (int)cudaGetLastError();
}

int hfx_dense_prove(const DevDB &db, const SpecMeta *meta, const BatchedWs &ws, const DenseWs &dw, const uint32_t *wb,
                    const uint32_t *we, const float *rows, int64_t stride, const float *kept_s,
                    const uint64_t *kept_k, int32_t nspec, int32_t topn, const float *out_s, const uint64_t *out_k,
                    SpecMeta *open_meta, uint32_t *n_open, cudaStream_t st) {
    if (topn > 32) return (int)cudaErrorInvalidValue;
    const cudaError_t e = cudaMemsetAsync(n_open, 0, 4, st);
    if (e != cudaSuccess) return (int)e;
    k_dense_ladders<<<dim3((unsigned)dw.cap_blocks, 64), 256, 0, st>>>(db.tc_sorted, db.tn_sorted, dw);
    k_dense_prove<<<(unsigned)((nspec + 3ll) / 4), 128, 0, st>>>(meta, ws.group_of, ws.groups, dw.blocks, wb, we, rows,
                                                                 stride, kept_s, kept_k, nspec, topn, out_s, out_k,
                                                                 open_meta, n_open);
    return (int)cudaGetLastError();
}

int hfx_dense_close(const SpecMeta *open_meta, const float *in_s, const uint64_t *in_k, int32_t nspec, int32_t topn,
                    const uint32_t *idx_sorted, float *out_s, uint64_t *out_k, uint32_t *out_pep, cudaStream_t st) {
    const int64_t n = (int64_t)nspec * topn;
    if (n <= 0) return 0;
    k_dense_close<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(open_meta, in_s, in_k, nspec, topn, idx_sorted, out_s,
                                                               out_k, out_pep);
    return (int)cudaGetLastError();
}
