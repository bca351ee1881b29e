// List-based batched scoring (the default batched path for unmodified
// candidates).
//
// Within one search step every candidate peptide is scored against many
// spectra (the +-tolerance windows of neighbouring spectra overlap).  So the
// step first builds, ONCE per (peptide, ion-charge level) that some spectrum
// of the batch needs, the ascending list of distinct ion bins with their
// intensity levels (ion_series.cu:78-123 with the max-dedupe of
// ion_series.cu:71-75), and stores it in HBM.  The scorer then streams a
// candidate's list -- entry i read by lane i % 32, which is exactly the
// canonical accumulation order -- and gathers the group tile in shared
// memory.  Nothing is reused across steps: the lists are rebuilt by every
// search.
//
// Which (peptide, level) pairs are needed: every spectrum adds its window
// [begin, end) to a difference array of its level; a prefix sum marks the
// covered peptides.
#include "hfx_internal.h"
#include "device_common.cuh"
#include "batched.h"
#include "lists.h"
#include "lists_device.cuh"
#include "scan.cuh"
#include <algorithm>
#include <type_traits>
#include "batched_common.cuh"

namespace hfx {

// ---- which (peptide, level) lists the batch needs ----
__global__ void k_mark_levels(const SpecMeta *__restrict__ meta, const uint32_t *__restrict__ wb,
                              const uint32_t *__restrict__ we, int32_t nspec, int64_t npep1,
                              int32_t *__restrict__ diff) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec) return;
    const SpecMeta m = meta[s];
    const int z = m.charges_plain;
    if (m.status != 0 || z < 1 || z > kLevels || we[s] <= wb[s]) return;
    atomicAdd(&diff[(int64_t)(z - 1) * npep1 + wb[s]], 1);
    atomicAdd(&diff[(int64_t)(z - 1) * npep1 + we[s]], -1);
}


// The candidates whose lists the batch needs, by class (entry: position |
// levels << 27), and the lengths of the lists it does not need.  One thread
// per peptide: a warp per peptide that looked at its coverage itself spent
// 0.18 ms on the 1.4 M peptides of the 20,000-protein database however few
// were needed.
constexpr int kNeedShift = 27;  // positions are below 2^27
__device__ __forceinline__ int long_class(uint32_t tc, uint32_t tn, uint32_t need);
template <bool kLong>
__global__ void __launch_bounds__(256) k_list_work(DevDB db, const int32_t *__restrict__ cover, int64_t npep1,
                                                   uint16_t *__restrict__ list_len, WorkLists wl,
                                                   uint32_t *__restrict__ err) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    int cls = -1;
    uint32_t need = 0;
    if (p < db.num_pep) {
#pragma unroll
        for (int z = 0; z < kLevels; ++z) {
            if (cover[(int64_t)z * npep1 + p] > 0) need |= 1u << z;
            else list_len[(size_t)z * db.num_pep + p] = 0;
        }
        if (need) {
            const uint32_t tc = db.tc_sorted[p], tn = db.tn_sorted[p];
            cls = kLong ? long_class(tc, tn, need) : list_class(tc, tn);
            if (cls < 0) {  // more keys than a warp sorts
                atomicOr(err, kErrTooLong);
                for (int z = 0; z < kLevels; ++z) list_len[(size_t)z * db.num_pep + p] = 0;
            }
        }
    }
    append_work(wl, cls, p | need << kNeedShift);
}

// The sorted distinct-bin list of every needed charge level of the candidates of
// one class, class_lanes lanes each (build_lists: the level-z list carries the
// level-(z-1) list over and adds the charge-z ions).  The 3.84 M lists (946 M
// entries) of 10,000 spectra against 20,000 proteins, coverage and work lists
// included: 4.12 ms by bit planes and a bit loop, 2.48 ms by rank with a warp each,
// 1.98 ms with two short ladders a warp.
template <bool FastDiv, int kClass>
__global__ void __launch_bounds__(256, kClass == 0 ? 1 : 4) k_gen_lists(DevDB db, int32_t nbins,
                                                                        const uint32_t *__restrict__ lstart,
                                                                        uint64_t total10, uint16_t *__restrict__ lists,
                                                                        uint16_t *__restrict__ list_len, WorkLists wl,
                                                                        unsigned long long *__restrict__ stats) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int W = class_lanes(kClass);
    const int lane = threadIdx.x & (W - 1), nw = blockDim.x / W;
    const RankBufs rb = rank_bufs(smem + (size_t)(threadIdx.x / W) * rank_bytes(nbins, kClass), nbins, kClass);
    __shared__ unsigned long long s_stats[3];
    if (threadIdx.x < 3) s_stats[threadIdx.x] = 0ull;
    for (int32_t i = lane; i < (rb.words >> 1); i += W) sts_u128(rb.pl + 16u * i, make_uint4(0u, 0u, 0u, 0u));
    __syncthreads();
    const float mt_lane = db.mt[threadIdx.x & 31];
    const uint32_t total = wl.count(kClass);
    const uint32_t *work = wl.list(kClass);
    uint32_t my_lists = 0, my_entries = 0, my_res = 0;
    for (uint32_t t = blockIdx.x * nw + threadIdx.x / W; (t & ~(32u / W - 1u)) < total; t += gridDim.x * nw) {
        // (a warp's last candidate may have no partner: no levels, no prefixes)
        const uint32_t w = t < total ? work[t] : 0u;
        const uint32_t p = w & ((1u << kNeedShift) - 1u), need = w >> kNeedShift;
        const uint32_t tc = db.tc_sorted[p], tn = need ? db.tn_sorted[p] : tc;
        // the slot holds 10 (tn - tc) z entries or more: every list fits
        const ListSlots ls{lists, total10, lstart[p], list_len + p, db.num_pep};
        const int entries = build_lists<FastDiv, kClass>(rb, db.ions, tc, tn, db.r_sorted[p], need, (uint32_t)nbins,
                                                         mt_lane, NoMods{}, ls);
        if (entries < 0) {
            if (lane == 0 && need) wl.list(0)[atomicAdd(wl.w, 1u)] = w;
            continue;
        }
        my_entries += (uint32_t)entries;
        my_lists += (uint32_t)__popc(need);
        my_res += tn > tc ? tn - tc : 0u;
    }
    if (stats) {
        if (lane == 0) {
            atomicAdd(&s_stats[0], (unsigned long long)my_lists);
            atomicAdd(&s_stats[1], (unsigned long long)my_entries);
            atomicAdd(&s_stats[2], (unsigned long long)my_res);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicAdd(&stats[0], s_stats[0]);
            atomicAdd(&stats[1], s_stats[1]);
            atomicAdd(&stats[6], s_stats[2]);
        }
    }
}

// ---- long rows: 32-bit list entries built by sorting ----
//
// With ~10^5 bins per row a bit per bin no longer fits in shared memory.
// Instead the warp writes the ten keys (bin, charge, level) of every (prefix,
// charge 1..zmax) of a needed peptide (ion_series.cu:78-123, the same
// arithmetic as item_bits) and sorts them once: a counting sort into up to 512
// ranges of bins (shared-memory counters, one scan, one scatter), then each
// key's place among the few keys of its range by comparing with them.  A key
// that opens a bin's run reads the run and has, for every charge level, the
// bin's highest level among the charges up to it -- the reference's atomicMax
// into the dense row (ion_series.cu:71-75) -- and ballots place it in the
// lists of the needed levels.
//
// What bounds it: shared-memory latency and instruction issue.  A bitonic sort
// per level with eight warps an SM (128 KB of keys) took 130 ms for the 4.2 M
// lists of a 10,000-spectrum batch at 0.02 Da; this takes 10.3 ms.
constexpr int kLongKeys = 4096;      // keys of a peptide that is accepted
constexpr int kLongRanges = 512;     // counting-sort ranges

// Class of a peptide by its keys: 1, 2 and 0 hold up to 1,024, 2,048 and
// kLongKeys keys (9, 18 and 34 KB of shared memory a warp); -1: too long.
__host__ __device__ constexpr int long_keys(int cls) { return cls == 1 ? 1024 : (cls == 2 ? 2048 : kLongKeys); }
__device__ __forceinline__ int long_class(uint32_t tc, uint32_t tn, uint32_t need) {
    if (tn < tc) return -1;
    const uint64_t n = 10ull * (tn - tc) * (uint32_t)(32 - __clz(need));
    return n <= 1024u ? 1 : (n <= 2048u ? 2 : (n <= (uint64_t)kLongKeys ? 0 : -1));
}
__host__ __device__ constexpr size_t long_bytes(int cls) { return (size_t)long_keys(cls) * 8 + kLongRanges * 4; }

// The bin rint(mz / d), y = RN(1 / d), for the mono or a custom width; from
// 2^31 on -- rows are shorter -- the uncorrected product, which keeps the
// conversion's saturation.
__device__ __forceinline__ uint32_t bin_long(float mz, float d, float y) {
    const float q = __fmul_rn(mz, y);
    return __float2uint_rz(q < 0x1p31f ? rintf(quotient(mz, d, y)) : q);
}

// A key holds the bin, the charge and the level, bin << 4 | (charge - 1) << 2 |
// level, of rows below 2^28 bins; in longer ones (kWide; a list entry holds 30
// bits of the bin) it has no charge, and every needed level is sorted by itself.
constexpr int32_t kNarrowBins = (1 << 28) - 1;

template <bool FastDiv, int kClass, bool kWide>
__global__ void __launch_bounds__(256) k_gen_lists_long(DevDB db, int32_t nbins, const uint32_t *__restrict__ lstart,
                                                        uint64_t total10, uint32_t *__restrict__ lists,
                                                        uint16_t *__restrict__ list_len, float width, WorkLists wl,
                                                        unsigned long long *__restrict__ stats) {
    constexpr int kBin = kWide ? 2 : 4;  // the key's bits below the bin
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t ka = smem_u32(smem) + (uint32_t)warp * (uint32_t)long_bytes(kClass);
    const uint32_t kb = ka + (uint32_t)long_keys(kClass) * 4u, cnt = kb + (uint32_t)long_keys(kClass) * 4u;
    __shared__ unsigned long long s_stats[3];
    if (threadIdx.x < 3) s_stats[threadIdx.x] = 0ull;
    __syncthreads();
    const float mt_lane = db.mt[lane];
    const float rwidth = __fdiv_rn(1.0f, width);
    // ranges of 2^shift bins
    int shift = 0;
    while ((nbins >> shift) >= kLongRanges) ++shift;
    const uint32_t total = wl.count(kClass);
    const uint32_t *work = wl.list(kClass);
    uint32_t my_lists = 0, my_entries = 0, my_res = 0;
    constexpr uint32_t kSteps = kWide ? kLevels : 1;  // of a candidate
    for (uint32_t t = blockIdx.x * nw + warp; t < total * kSteps; t += gridDim.x * nw) {
        const uint32_t w = work[t / kSteps];
        const uint32_t p = w & ((1u << kNeedShift) - 1u);
        const uint32_t need = kWide ? (w >> kNeedShift) & (1u << (t % kSteps)) : w >> kNeedShift;
        if (kWide && !need) continue;
        const int zmax = 32 - __clz(need);
        const uint32_t tc = db.tc_sorted[p];
        const int len = (int)(db.tn_sorted[p] - tc);
        const float residual = db.r_sorted[p];
        const uint32_t slot = lstart[p];
        my_res += kWide && ((w >> kNeedShift) & (need - 1u)) ? 0u : (uint32_t)len;
#pragma unroll
        for (int i = 0; i < kLongRanges / 128; ++i) sts_u128(cnt + 16u * (uint32_t)(32 * i + lane), make_uint4(0u, 0u, 0u, 0u));
        __syncwarp();
        // the keys (~0: outside the row), charge by charge, and how many fall
        // into each range
        float carry = 0.0f;
        for (int k0 = 0; k0 < len; k0 += 32) {
            NoMods mods;
            const int c32 = min(32, len - k0);
            const float b = ladder_chunk(db.ions, tc + (uint32_t)k0, c32, mt_lane, mods, carry);
            carry = __shfl_sync(kFullMask, b, c32 - 1);
            const float y = __fsub_rn(residual, b);
#pragma unroll 1
            for (int z = 1; z <= zmax; ++z) {
                const ChargeConst kc = charge_const<FastDiv>(z);
                auto bin = [&](float mz) -> uint32_t {
                    if constexpr (FastDiv) return (uint32_t)sat_bin(rintf(__fdividef(mz, width)));
                    else return bin_long(mz, width, rwidth);
                };
                const float mb = div_charge<FastDiv>(__fadd_rn(b, kc.hc), z);
                const float my = div_charge<FastDiv>(__fadd_rn(__fadd_rn(y, kH2O), kc.hc), z);
                const uint32_t xb = bin(mb), xy = bin(my);
                const uint32_t x[10] = {bin(div_charge<FastDiv>(__fadd_rn(__fsub_rn(b, kCO), kc.hc), z)),
                                        bin(__fsub_rn(mb, kc.dh2o)),
                                        bin(__fsub_rn(mb, kc.dnh3)),
                                        bin(__fsub_rn(my, kc.dnh3)),
                                        xb - 1u, xb + 1u, xy - 1u, xy + 1u, xb, xy};
                const uint32_t at = ka + 40u * (uint32_t)((z - 1) * len + k0 + lane);
                if (lane < c32) {
#pragma unroll
                    for (int j = 0; j < 10; ++j) {
                        const bool in = x[j] < (uint32_t)nbins;
                        const uint32_t key = x[j] << kBin | (kWide ? 0u : (uint32_t)(z - 1) << 2) |
                                             (j < 4 ? 1u : (j < 8 ? 2u : 3u));
                        sts_u32(at + 4u * j, in ? key : ~0u);
                        if (in) red_add(cnt + 4u * (x[j] >> shift), 1u);
                    }
                }
            }
        }
        __syncwarp();
        // starts of the ranges
        uint32_t n = 0;
#pragma unroll 1
        for (int i = 0; i < kLongRanges / 128; ++i) {
            const uint32_t at = cnt + 16u * (uint32_t)(32 * i + lane);
            const uint4 c = lds_u128(at);
            const uint32_t own = c.x + c.y + c.z + c.w;
            const uint32_t incl = (uint32_t)warp_incl_scan((int)own);
            const uint32_t e = n + incl - own;
            sts_u128(at, make_uint4(e, e + c.x, e + c.x + c.y, e + c.x + c.y + c.z));
            n += __shfl_sync(kFullMask, incl, 31);
        }
        __syncwarp();
        // scatter; a range's counter ends at its end
        const int raw = 10 * len * zmax;
#pragma unroll 1
        for (int i = lane; i < raw; i += 32) {
            const uint32_t k = lds_u32(ka + 4u * i);
            if (k != ~0u) sts_u32(kb + 4u * atom_add(cnt + 4u * (k >> (kBin + shift)), 1u), k);
        }
        __syncwarp();
        // each key's place within its range
#pragma unroll 1
        for (int i = lane; i < (int)n; i += 32) {
            const uint32_t k = lds_u32(kb + 4u * i);
            const uint32_t r = k >> (kBin + shift);
            uint32_t at = r ? lds_u32(cnt + 4u * r - 4u) : 0u;
            const uint32_t end = lds_u32(cnt + 4u * r);
            uint32_t place = at;
            for (; at < end; ++at) {
                const uint32_t o = lds_u32(kb + 4u * at);
                place += (o < k || (o == k && at < (uint32_t)i)) ? 1u : 0u;
            }
            sts_u32(ka + 4u * place, k);
        }
        __syncwarp();
        // the runs of equal bins; byte z - 1 of `best`: the highest level up to charge z
        uint32_t out_n[kLevels];
#pragma unroll
        for (int z = 0; z < kLevels; ++z) out_n[z] = 0u;
#pragma unroll 1
        for (int i0 = 0; i0 < (int)n; i0 += 32) {
            const int i = i0 + lane;
            uint32_t best = 0u, bin = ~0u;
            if (i < (int)n) {
                const uint32_t k = lds_u32(ka + 4u * i);
                bin = k >> kBin;
                if (i == 0 || (lds_u32(ka + 4u * i - 4u) >> kBin) != bin) {
                    uint32_t o = k;
                    for (int j = i;;) {
                        const uint32_t c = kWide ? 0u : (o >> 2) & 3u;
                        best = __vmaxu4(best, ((o & 3u) * 0x01010101u) << (8u * c));
                        if (++j >= (int)n) break;
                        o = lds_u32(ka + 4u * j);
                        if ((o >> kBin) != bin) break;
                    }
                }
            }
#pragma unroll
            for (int z = 0; z < kLevels; ++z) {
                if (!((need >> z) & 1u)) continue;
                const uint32_t lvl = (best >> (8 * z)) & 0xFFu;
                const uint32_t bal = __ballot_sync(kFullMask, lvl != 0u);
                if (lvl)
                    lists[total10 * (uint64_t)(z * (z + 1) / 2) + (uint64_t)(z + 1) * slot + out_n[z] +
                          (uint32_t)__popc(bal & ((1u << lane) - 1u))] = bin << 2 | lvl;
                out_n[z] += (uint32_t)__popc(bal);
            }
        }
#pragma unroll
        for (int z = 0; z < kLevels; ++z)
            if ((need >> z) & 1u) {
                if (lane == 0) list_len[(size_t)z * db.num_pep + p] = (uint16_t)out_n[z];
                my_lists += 1u;
                my_entries += out_n[z];
            }
        __syncwarp();
    }
    if (stats) {
        if (lane == 0) {
            atomicAdd(&s_stats[0], (unsigned long long)my_lists);
            atomicAdd(&s_stats[1], (unsigned long long)my_entries);
            atomicAdd(&s_stats[2], (unsigned long long)my_res);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicAdd(&stats[0], s_stats[0]);
            atomicAdd(&stats[1], s_stats[1]);
            atomicAdd(&stats[6], s_stats[2]);
        }
    }
}

// FP32 rescoring of kept unmodified candidates from their lists and the
// FP32 row in global memory (long rows), canonical order: entry i by lane
// i % 32, XOR butterfly.  One CTA per spectrum.
template <typename E>
__global__ void __launch_bounds__(256) k_rescore_lists(const E *__restrict__ lists,
                                                       const uint32_t *__restrict__ lstart, uint64_t total10,
                                                       const uint16_t *__restrict__ list_len, uint32_t num_pep,
                                                       const uint32_t *__restrict__ idx_sorted,
                                                       const float *__restrict__ rows32, int64_t stride,
                                                       const SpecMeta *__restrict__ meta,
                                                       const uint64_t *__restrict__ kept_k, int32_t K, int32_t topn,
                                                       float *__restrict__ out_s, uint64_t *__restrict__ out_k,
                                                       uint32_t *__restrict__ out_pep, uint32_t *__restrict__ err) {
    __shared__ float res_s[kMaxKept];
    __shared__ uint64_t res_k[kMaxKept];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t s = blockIdx.x;
    const SpecMeta m = meta[s];
    const float *row = rows32 + (size_t)s * stride;
    const int z = m.charges_plain;
    for (int t = warp; t < K; t += nw) {
        const uint64_t kk = kept_k[(size_t)s * K + t];
        float sc = -INFINITY;
        if (kk != ~0ull) {
            float acc = 0.0f;
            if (!(kk >> 63) && z >= 1 && kk < num_pep) {
                const uint32_t p = (uint32_t)kk;
                const int n = list_len[(size_t)(z - 1) * num_pep + p];
                const E *lp = lists + list_offset(lstart, total10, z, p);
                // four entries per lane in flight, then their row values,
                // then the sums in the lane's ascending entry order
                for (int i0 = lane; i0 < n; i0 += 128) {
                    uint32_t e[4];
                    float x[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) e[k] = i0 + 32 * k < n ? (uint32_t)__ldg(lp + i0 + 32 * k) : ~0u;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t bin = e[k] >> 2;
                        x[k] = (i0 + 32 * k < n && (int32_t)bin < m.len) ? __ldg(row + bin) : 0.0f;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (i0 + 32 * k < n && (int32_t)(e[k] >> 2) < m.len)
                            acc = __fmaf_rn(level_weight(e[k] & 3u), x[k], acc);
                }
            } else if (kk >> 63) {
                if (lane == 0) atomicOr(err, kErrBounds);
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(kFullMask, acc, o));
            sc = acc;
        }
        if (lane == 0) {
            res_s[t] = sc;
            res_k[t] = kk;
        }
    }
    __syncthreads();
    if (warp == 0) {
        WarpTopK tk;
        tk.init();
        for (int t = 0; t < K; ++t)
            if (res_k[t] != ~0ull) tk.insert(res_s[t], res_k[t], topn);
        if (lane < topn) {
            out_s[(size_t)s * topn + lane] = tk.s;
            out_k[(size_t)s * topn + lane] = tk.k;
            out_pep[(size_t)s * topn + lane] = (tk.k != ~0ull && tk.k < num_pep) ? idx_sorted[tk.k] : ~0u;
        }
    }
}

// Scorer over precomputed lists: a persistent grid pulls work items (group x
// candidate chunk); the group's interleaved tile is staged by one bulk copy;
// a warp streams each candidate's list (entry i by lane i % 32, four loads
// in flight per lane) and gathers the tile; CTA-wide top-K per member.
// E = list entry type (uint16_t up to 16,383 bins, uint32_t for long rows);
// kGlobal: the group tile is read from global memory (L2) instead of being
// staged in shared memory (rows too long for shared memory).
// kC: candidates per warp (1, 2 or 4), one per group of 32 / kC lanes (entry
// i of a list by lane i % (32 / kC) of its group).  The per-candidate work
// around the list -- the claim, the reduction, the admission -- is then
// shared by kC candidates.  In FP32 with four candidates each lane keeps four
// partial-sum sets (entry k of every round of 32 in set k) and adds them as
// the 32-lane butterfly would, so the sums keep the canonical order; the
// BF16/FP16 pass sums in one set (its scores only pick the candidates that
// FP32 rescoring orders).
template <typename T, int G, typename E, bool kGlobal, int kC, int L>
__global__ void __launch_bounds__(1024, 1)
k_score_lists(const E *__restrict__ lists, const uint32_t *__restrict__ lstart, uint64_t total10,
              uint64_t list_total, const uint16_t *__restrict__ list_len, uint32_t num_pep,
              const T *__restrict__ tiles, int64_t stride,
              const uint32_t *__restrict__ wb, const uint32_t *__restrict__ we, const int32_t *__restrict__ perm,
              const GroupInfo *__restrict__ groups, const uint32_t *__restrict__ item_off,
              const uint32_t *__restrict__ ngroups_p, int32_t K, uint32_t *__restrict__ counter,
              float *__restrict__ part_s, uint64_t *__restrict__ part_k, unsigned long long *__restrict__ stats,
              float *__restrict__ sink, const uint64_t *__restrict__ sink_off, uint32_t qoff,
              uint32_t *__restrict__ err) {
    static_assert(kC == 1 || kC == 2 || kC == 4, "1, 2 or 4 candidates per warp");
    constexpr int kW = 32 / kC;  // lanes per candidate
    // FP32 with several candidates per warp: four partial-sum sets per lane
    constexpr bool kSets4 = std::is_same<T, float>::value && kC > 1;
    static_assert(!kSets4 || kW == 8, "the FP32 partial-sum sets assume 8 lanes per candidate");
    static_assert(G <= kW, "a lane group takes up to one spectrum of the group per lane");
    using Entries = EntryRound<E, kW>;
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int hl = lane & (kW - 1), half = lane / kW;  // `half`: the lane's candidate group
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    T *stile = reinterpret_cast<T *>(smem + 128);
    const T *tile = stile;
    __shared__ int32_t s_item;
    __shared__ uint32_t s_next;
    __shared__ uint32_t s_wb[G], s_we[G];
    __shared__ uint64_t s_off[G];  // with a sink: where each member's window starts in it
    __shared__ uint32_t thr_u[G], s_lock[G];
    __shared__ float s_ls[G * L];
    __shared__ uint32_t s_lk[G * L];
    __shared__ unsigned long long s_stats[5];

    const int32_t ngroups = (int32_t)*ngroups_p;
    const uint32_t total = item_off[ngroups];
    if (threadIdx.x == 0) mbar_init(bar, 1);
    if (threadIdx.x < 5) s_stats[threadIdx.x] = 0ull;
    __syncthreads();
    const int my_slot = reduce_slot_of_lane<G>(lane);
    uint32_t my_cand = 0, my_entries = 0, my_psm = 0, my_claims = 0;
    uint32_t phase = 0;
    CtaSlots<G, uint32_t, cta_queue_len(G), L> slots;
    slots.bind(s_ls, s_lk, s_lock, thr_u, smem + qoff + (size_t)warp * CtaSlots<G>::warp_bytes(), err);
    while (true) {
        if (threadIdx.x == 0) s_item = (int32_t)atomicAdd(counter, 1u);
        __syncthreads();
        const uint32_t item = (uint32_t)s_item;
        if (item >= total) break;
        const int32_t g = find_group(item_off, ngroups, item);
        const GroupInfo gi = groups[g];
        const uint32_t p0 = gi.lo + (item - item_off[g]) * gi.chunk;
        const uint32_t p1 = min(gi.hi, p0 + gi.chunk);
        const int cnt_members = (int)gi.count;
        if (threadIdx.x < G) {
            const int j = threadIdx.x;
            uint32_t b = 0, e = 0;
            uint64_t o = 0;
            if (j < cnt_members) {
                const int32_t s = perm[gi.pos0 + j];
                b = wb[s];
                e = we[s];
                if (sink) o = sink_off[s];
            }
            s_off[j] = o;
            s_wb[j] = b;
            s_we[j] = e;
        }
        slots.reset_shared();
        const int32_t nb = tile_bins(gi.maxlen);
        if (threadIdx.x == 0) {
            s_next = p0;
            my_claims += p1 - p0;
            if (stats && !kGlobal) s_stats[4] += (unsigned long long)nb * G * sizeof(T);
        }
        if constexpr (kGlobal) {
            tile = tiles + (size_t)g * stride * G;
            __syncthreads();
        } else {
            if (threadIdx.x == 0) {
                fence_proxy_async();
                const uint32_t bytes = (uint32_t)((size_t)nb * G * sizeof(T));
                mbar_arrive_expect_tx(bar, bytes);
                bulk_g2s(stile, tiles + (size_t)g * stride * G, bytes, bar);
            }
            // bins [nb, stride + 8) of the shared tile read as zero: every
            // list bin (< stride) and the pad entry (bin = stride) may be
            // gathered without a bounds test
            {
                uint4 *z = reinterpret_cast<uint4 *>(stile);
                const size_t z0 = (size_t)nb * G * sizeof(T) / 16, z1 = (size_t)(stride + 8) * G * sizeof(T) / 16;
                for (size_t i = z0 + threadIdx.x; i < z1; i += blockDim.x) z[i] = make_uint4(0u, 0u, 0u, 0u);
                fence_proxy_async();  // before a later item's bulk copy overwrites these bytes
            }
            __syncthreads();
            if (!mbar_wait(bar, phase, kWaitLimit)) {
                if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
                return;
            }
            phase ^= 1u;
        }
        // member hl's window, in each half
        const uint32_t my_b = hl < G ? s_wb[hl] : 0u, my_e = hl < G ? s_we[hl] : 0u;
        // entry past a list's end: the zero bin `stride` of the shared tile
        // (beyond every group's bins, so it also ends the scan), or an
        // out-of-range bin for tiles in global memory
        const uint32_t pad = kGlobal ? 0xFFFFFFFFu : ((uint32_t)stride << 2);
        const int z = (int)gi.charges;
        const uint16_t *llen = list_len + (size_t)(z >= 1 ? z - 1 : 0) * num_pep;
        // Three-stage software pipeline over the warp's candidates: while
        // candidate i is scored, candidate i+1's first list entries are in
        // flight and candidate i+2 is claimed with its list length and
        // offset loads in flight, so no stage waits on a dependent load.
        // Per lane: its half's candidate; `live` (warp-uniform) while any
        // candidate was claimed.
        struct Meta {
            uint32_t p, act, n, ls;
            bool live;
        };
        struct Cand {
            uint32_t p, act;
            int n;
            bool live;
            const E *lp;
            Entries e;
        };
        auto claim = [&]() {
            Meta m;
            m.act = 0u;
            m.n = 0u;
            m.ls = 0u;
            while (true) {
                uint32_t q = 0;
                if (lane == 0) q = atomicAdd(&s_next, (uint32_t)kC);
                const uint32_t base = __shfl_sync(kFullMask, q, 0);
                m.live = base < p1;
                m.p = base + (uint32_t)half;
                if (!m.live) break;
                const uint32_t bal =
                    __ballot_sync(kFullMask, hl < G && m.p < p1 && my_b <= m.p && m.p < my_e);
                m.act = (bal >> (kW * half)) & ((1u << G) - 1u);
                if (bal) break;
            }
            if (m.act && z >= 1 && m.p < num_pep) {
                m.n = llen[m.p];
                m.ls = lstart[m.p];
            }
            return m;
        };
        auto issue = [&](const Meta &m) {
            Cand c;
            c.p = m.p;
            c.act = m.act;
            c.n = (int)m.n;
            c.live = m.live;
            c.lp = lists;
            if (m.act && z >= 1) {
                const uint64_t off = total10 * (uint64_t)(z * (z - 1) / 2) + (uint64_t)z * m.ls;
                if (m.p >= num_pep || off + (uint64_t)c.n > list_total) {
                    if (hl == 0) atomicOr(err, kErrBounds);
                    c.n = 0;
                } else {
                    c.lp = lists + off;
                }
            }
            c.e.load(c.lp, 0, hl, c.n, pad);
            return c;
        };
        Meta ahead = claim();
        Cand nxt = issue(ahead);
        if (nxt.live) ahead = claim();
        while (nxt.live) {
            const Cand cur = nxt;
            nxt = issue(ahead);
            if (nxt.live) ahead = claim();
            float acc[G];
#pragma unroll
            for (int j = 0; j < G; ++j) acc[j] = 0.0f;
            // FP32 with four candidates per warp keeps the canonical order:
            // entry i of a list goes to partial sum i % 32, and with 8 lanes
            // per candidate entry k of each round of 32 is partial 8 k + lane,
            // so each lane keeps four partial-sum sets and adds them as the
            // 32-lane butterfly's offsets 16 and 8 do
            float acc4[kSets4 ? 4 : 1][G];
#pragma unroll
            for (int k = 0; k < (kSets4 ? 4 : 1); ++k)
#pragma unroll
                for (int j = 0; j < G; ++j) acc4[k][j] = 0.0f;
            const int n = cur.n;
            int nmax = n;
#pragma unroll
            for (int o = kW; o < 32; o <<= 1) nmax = max(nmax, __shfl_xor_sync(kFullMask, nmax, o));
            // entries [i0, i0 + 4 kW) in e, the next 4 kW already in flight in f
            Entries e = cur.e, f;
            f.load(cur.lp, 4 * kW, hl, n, pad);
            for (int i0 = 0; i0 < nmax; i0 += 4 * kW) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t w = e.e[k], bin = w >> 2;
                    float *a = acc;
                    if constexpr (kSets4) a = acc4[k];
                    if constexpr (kGlobal) {
                        if ((int32_t)bin < nb)
                            TileFma<T, G>::fma(tile, bin, w & 3u, *reinterpret_cast<float(*)[G]>(a));
                    } else {
                        // zero beyond nb
                        TileFma<T, G>::fma(tile, bin, w & 3u, *reinterpret_cast<float(*)[G]>(a));
                    }
                }
                // lists ascend: once an entry lies beyond the tile, so do the rest
                const uint32_t last = __shfl_sync(kFullMask, e.e[3], (lane & ~(kW - 1)) | (kW - 1));
                if (__all_sync(kFullMask, (last >> 2) >= (uint32_t)nb)) break;
                e = f;
                f.load(cur.lp, i0 + 8 * kW, hl, n, pad);
            }
            if constexpr (kSets4) {
                // offsets 16 (partials l and l + 16, l + 8 and l + 24) and 8
#pragma unroll
                for (int j = 0; j < G; ++j)
                    acc[j] = __fadd_rn(__fadd_rn(acc4[0][j], acc4[2][j]), __fadd_rn(acc4[1][j], acc4[3][j]));
            }
            if constexpr (kC > 1) {
                const float sc = reduce_scatter_lanes<G, kW>(acc);
                if (hl == 0 && cur.act) {
                    my_cand += 1u;
                    my_entries += (uint32_t)n;
                    my_psm += (uint32_t)__popc(cur.act);
                }
                // lane j * kW / G of a candidate's lanes has member j's score
                const int mine = hl / (kW / G);
                const bool holds = (hl & (kW / G - 1)) == 0 && ((cur.act >> mine) & 1u);
                // every pair's score, at its member's window offset
                // (E-values; FP32 only, the host refuses a sink otherwise)
                if constexpr (std::is_same<T, float>::value) {
                    if (sink && holds) sink[s_off[mine] + (cur.p - s_wb[mine])] = sc;
                }
                // the queues take the four when one beats its list's last
                if (!__any_sync(kFullMask, holds && score_order(sc) >= *(volatile uint32_t *)(thr_u + mine))) continue;
                const bool owner = (lane & (32 / G - 1)) == 0;
#pragma unroll
                for (int q = 0; q < kC; ++q) {
                    const uint32_t act_q = __shfl_sync(kFullMask, cur.act, q * kW);
                    const uint32_t p_q = __shfl_sync(kFullMask, cur.p, q * kW);
                    // member j's admission lane is j * 32 / G
                    const float sc_q = __shfl_sync(kFullMask, sc, q * kW + (lane / (32 / G)) * (kW / G));
                    const bool want = owner && ((act_q >> my_slot) & 1u) &&
                                      score_order(sc_q) >= *(volatile uint32_t *)(thr_u + my_slot);
                    slots.offer(want, sc_q, p_q, my_slot, K);
                }
            } else {
                if (lane == 0) {
                    my_cand += 1u;
                    my_entries += (uint32_t)n;
                    my_psm += (uint32_t)__popc(cur.act);
                }
                const float sc = reduce_scatter<G>(acc);
                if (sink) {
                    // every pair's score, at its member's window offset (the
                    // admission below still keeps the top-K)
                    if ((lane & (32 / G - 1)) == 0 && ((cur.act >> my_slot) & 1u))
                        sink[s_off[my_slot] + (cur.p - s_wb[my_slot])] = sc;
                }
                const bool want = (lane & (32 / G - 1)) == 0 && ((cur.act >> my_slot) & 1u) &&
                                  score_order(sc) >= *(volatile uint32_t *)(thr_u + my_slot);
                slots.offer(want, sc, cur.p, my_slot, K);
            }
        }
        slots.drain(K);
        __syncthreads();  // every warp has merged its queues
        for (int j = warp; j < cnt_members; j += nw) {
            const size_t o = ((size_t)item * G + j) * K;
            slots.result(j, K, part_s + o, part_k + o);
        }
        __syncthreads();
    }
    if (stats) {
        if (hl == 0) {
            atomicAdd(&s_stats[0], (unsigned long long)my_cand);
            atomicAdd(&s_stats[1], (unsigned long long)my_entries);
            atomicAdd(&s_stats[2], (unsigned long long)my_psm);
            atomicAdd(&s_stats[3], (unsigned long long)my_claims);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicAdd(&stats[2], s_stats[0]);
            atomicAdd(&stats[3], s_stats[1]);
            atomicAdd(&stats[4], s_stats[2]);
            atomicAdd(&stats[5], s_stats[3]);
            atomicAdd(&stats[7], s_stats[4]);
        }
    }
}

}  // namespace hfx

using namespace hfx;

int hfx_scan_inclusive(const int32_t *in, int64_t n, int32_t *out, int32_t *partial, cudaStream_t st) {
    return scan_inclusive<int32_t>(in, n, out, partial, st);
}

int64_t hfx_scan_partials_needed(int64_t n) { return scan_partials<int32_t>(n); }

int hfx_lists_mark(const SpecMeta *meta, const uint32_t *wb, const uint32_t *we, int32_t nspec, int64_t npep1,
                   int32_t *diff, cudaStream_t st) {
    cudaMemsetAsync(diff, 0, sizeof(int32_t) * (size_t)kLevels * npep1, st);
    if (nspec > 0) k_mark_levels<<<(nspec + 255) / 256, 256, 0, st>>>(meta, wb, we, nspec, npep1, diff);
    return (int)cudaGetLastError();
}

size_t hfx_lists_work_words(uint64_t n) { return work_words(n); }
uint64_t hfx_lists_work_cap(uint64_t words) { return words > work_words(0) ? (words - work_words(0)) / kWorkLists : 0; }

int hfx_lists_generate(const DevDB &db, const int32_t *cover, int64_t npep1, int32_t nbins, const uint32_t *lstart,
                       uint64_t total10, uint16_t *lists, uint16_t *list_len, uint32_t *work, int fastdiv,
                       unsigned long long *stats, cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const WorkLists wl{work, db.num_pep};
    cudaMemsetAsync(work, 0, 16, st);
    k_list_work<false><<<(db.num_pep + 255) / 256, 256, 0, st>>>(db, cover, npep1, list_len, wl, nullptr);
    auto run = [&](auto f, int cls) {
        const size_t smem = (size_t)(256 / class_lanes(cls)) * rank_bytes(nbins, cls);
        // the limit is the function's, common to all contexts and threads: that of the longest rows
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((256 / class_lanes(cls)) * rank_bytes(kMaxWords * 32, cls)));
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, 256, smem);
        f<<<sms * std::max(1, cls ? per : std::min(per, 2)), 256, smem, st>>>(db, nbins, lstart, total10, lists,
                                                                             list_len, wl, stats);
    };
    run(fastdiv ? k_gen_lists<true, 3> : k_gen_lists<false, 3>, 3);
    run(fastdiv ? k_gen_lists<true, 1> : k_gen_lists<false, 1>, 1);
    run(fastdiv ? k_gen_lists<true, 2> : k_gen_lists<false, 2>, 2);
    run(fastdiv ? k_gen_lists<true, 0> : k_gen_lists<false, 0>, 0);
    return (int)cudaGetLastError();
}

// Candidates per warp with groups of up to 8 spectra (FP32 and BF16/FP16).
constexpr int kLowpCands = 4;

// Warps per list-scorer CTA: 16 (two CTAs per SM) up to 8 spectra per
// group, 32 (one CTA per SM, the tile taking most of shared memory) for 16.
constexpr int list_warps(int G) { return G >= 16 ? 32 : 16; }

// Dynamic shared memory of the list scorer: an mbarrier, the group tile
// (none when it is read from global memory), then the warps' queues.
static size_t lists_queue_offset(bool global_tile, int64_t stride, int G, size_t elem_bytes) {
    // the shared tile holds stride + 8 bins: the zero bins after the group's
    // rows and the pad entry's bin
    return 128 + (global_tile ? 0 : (((size_t)(stride + 8) * G * elem_bytes + 15) & ~(size_t)15));
}

template <typename T, int G, typename E, bool kGlobal, int kC, int L>
static int launch_lists_t(const E *lists, const uint32_t *lstart, uint64_t total10, const uint16_t *list_len,
                          uint32_t num_pep, int64_t stride, const uint32_t *wb, const uint32_t *we,
                          const BatchedWs &ws, void *tiles, int32_t K, int nw,
                          float *part_s, uint64_t *part_k, unsigned long long *stats, float *sink,
                          const uint64_t *sink_off, uint32_t *err, cudaStream_t st) {
    int dev = 0, sms = 0, smem_max = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (nw <= 0) nw = list_warps(G);
    const size_t qoff = lists_queue_offset(kGlobal, stride, G, sizeof(T));
    const size_t smem = qoff + (size_t)nw * CtaSlots<G>::warp_bytes();
    if (smem > (size_t)smem_max) return (int)cudaErrorInvalidValue;
    auto fn = k_score_lists<T, G, E, kGlobal, kC, L>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, nw * 32, smem);
    const int grid = sms * (per > 0 ? per : 1);
    cudaMemsetAsync(ws.counter, 0, 4, st);
    fn<<<grid, nw * 32, smem, st>>>(lists, lstart, total10, total10 * 10, list_len, num_pep, (const T *)tiles,
                                    stride, wb, we, ws.perm, ws.groups, ws.item_off, ws.ngroups, K,
                                    ws.counter, part_s, part_k, stats, sink, sink_off, (uint32_t)qoff, err);
    return (int)cudaGetLastError();
}

int hfx_lists_group_fits(int32_t G, int long_rows, int64_t stride, int elem_bytes) {
    if (G != 16) return 1;
    int dev = 0, smem_max = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    const cudaError_t e =
        long_rows ? cudaFuncGetAttributes(&fa, k_score_lists<__nv_bfloat16, 16, uint32_t, true, 1, 32>)
                  : cudaFuncGetAttributes(&fa, k_score_lists<__nv_bfloat16, 16, uint16_t, false, 1, 32>);
    if (e != cudaSuccess) return 0;
    const size_t smem = lists_queue_offset(long_rows != 0, stride, 16, (size_t)elem_bytes) +
                        (size_t)list_warps(16) * CtaSlots<16>::warp_bytes();
    return smem + fa.sharedSizeBytes <= (size_t)smem_max ? 1 : 0;
}

int hfx_lists_score(const void *lists, int long_rows, const uint32_t *lstart, uint64_t total10,
                    const uint16_t *list_len, uint32_t num_pep, int elem_kind, int64_t stride, const uint32_t *wb,
                    const uint32_t *we, const BatchedWs &ws, void *tiles, int32_t G, int32_t K, int nw,
                    float *part_s, uint64_t *part_k, unsigned long long *stats, uint32_t *err, cudaStream_t st,
                    float *sink, const uint64_t *sink_off) {
    // groups of up to 8 spectra score four candidates per warp (FP32 in the
    // canonical order, with or without a sink; BF16/FP16 scores only choose
    // what FP32 rescoring orders)
    if (elem_kind != 0 && sink) return (int)cudaErrorInvalidValue;
    // up to 64 kept candidates per member in the BF16/FP16 pass
    if (K > kMaxKept || (K > 32 && (elem_kind == 0 || G > 8))) return (int)cudaErrorInvalidValue;
#define HFX_LL(T, GG, LL)                                                                                      \
    do {                                                                                                       \
        constexpr int kP = GG > 8 ? 1 : kLowpCands;                                                            \
        if (long_rows)                                                                                         \
            return launch_lists_t<T, GG, uint32_t, true, kP, LL>((const uint32_t *)lists, lstart, total10,     \
                                                                 list_len, num_pep, stride, wb, we, ws, tiles, \
                                                                 K, nw, part_s, part_k, stats, sink, sink_off, \
                                                                 err, st);                                     \
        return launch_lists_t<T, GG, uint16_t, false, kP, LL>((const uint16_t *)lists, lstart, total10,        \
                                                              list_len, num_pep, stride, wb, we, ws, tiles, K, \
                                                              nw, part_s, part_k, stats, sink, sink_off, err,  \
                                                              st);                                             \
    } while (0)
#define HFX_L(T, GG) HFX_LL(T, GG, 32)
#define HFX_L64(T, GG)                 \
    do {                               \
        if (K > 32) HFX_LL(T, GG, 64); \
        HFX_LL(T, GG, 32);             \
    } while (0)
    if (elem_kind == 0) {
        if (G == 4) HFX_L(float, 4);
        if (G == 8) HFX_L(float, 8);
        if (G == 2) HFX_L(float, 2);
        if (G == 1) HFX_L(float, 1);
    } else if (elem_kind == 1) {
        if (G == 8) HFX_L64(__nv_bfloat16, 8);
        if (G == 16) HFX_L(__nv_bfloat16, 16);
        if (G == 4) HFX_L64(__nv_bfloat16, 4);
        if (G == 2) HFX_L64(__nv_bfloat16, 2);
        if (G == 1) HFX_L64(__nv_bfloat16, 1);
    } else {
        if (G == 8) HFX_L64(__half, 8);
        if (G == 16) HFX_L(__half, 16);
        if (G == 4) HFX_L64(__half, 4);
        if (G == 2) HFX_L64(__half, 2);
        if (G == 1) HFX_L64(__half, 1);
    }
#undef HFX_L64
#undef HFX_LL
#undef HFX_L
    return (int)cudaErrorInvalidValue;
}

int hfx_lists_generate_long(const DevDB &db, const int32_t *cover, int64_t npep1, int32_t nbins,
                            const uint32_t *lstart, uint64_t total10, uint32_t *lists, uint16_t *list_len,
                            uint32_t *work, int fastdiv, float ion_bw, unsigned long long *stats, uint32_t *err,
                            cudaStream_t st) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const WorkLists wl{work, db.num_pep};
    cudaMemsetAsync(work, 0, 16, st);
    k_list_work<true><<<(db.num_pep + 255) / 256, 256, 0, st>>>(db, cover, npep1, list_len, wl, err);
    const float width = ion_bw > 0.0f ? ion_bw : kBinMono;
    auto run = [&](auto f, int cls, int nw) {
        const size_t smem = (size_t)nw * long_bytes(cls);
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, nw * 32, smem);
        f<<<sms * std::max(1, per), nw * 32, smem, st>>>(db, nbins, lstart, total10, lists, list_len, width, wl,
                                                         stats);
    };
    if (nbins <= kNarrowBins) {
        run(fastdiv ? k_gen_lists_long<true, 1, false> : k_gen_lists_long<false, 1, false>, 1, 8);
        run(fastdiv ? k_gen_lists_long<true, 2, false> : k_gen_lists_long<false, 2, false>, 2, 4);
        run(fastdiv ? k_gen_lists_long<true, 0, false> : k_gen_lists_long<false, 0, false>, 0, 2);
    } else {
        run(fastdiv ? k_gen_lists_long<true, 1, true> : k_gen_lists_long<false, 1, true>, 1, 8);
        run(fastdiv ? k_gen_lists_long<true, 2, true> : k_gen_lists_long<false, 2, true>, 2, 4);
        run(fastdiv ? k_gen_lists_long<true, 0, true> : k_gen_lists_long<false, 0, true>, 0, 2);
    }
    return (int)cudaGetLastError();
}

int hfx_rescore_lists(const void *lists, int long_rows, const uint32_t *lstart, uint64_t total10,
                      const uint16_t *list_len, uint32_t num_pep, const uint32_t *idx_sorted, const float *rows32,
                      int64_t stride, const SpecMeta *meta, const uint64_t *kept_k, int32_t nspec, int32_t K,
                      int32_t topn, float *out_s, uint64_t *out_k, uint32_t *out_pep, uint32_t *err,
                      cudaStream_t st) {
    if (nspec <= 0) return 0;
    if (long_rows)
        k_rescore_lists<uint32_t><<<nspec, 256, 0, st>>>((const uint32_t *)lists, lstart, total10, list_len, num_pep,
                                                         idx_sorted, rows32, stride, meta, kept_k, K, topn, out_s,
                                                         out_k, out_pep, err);
    else
        k_rescore_lists<uint16_t><<<nspec, 256, 0, st>>>((const uint16_t *)lists, lstart, total10, list_len, num_pep,
                                                         idx_sorted, rows32, stride, meta, kept_k, K, topn, out_s,
                                                         out_k, out_pep, err);
    return (int)cudaGetLastError();
}
