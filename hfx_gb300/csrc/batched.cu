// Batched search: every spectrum of a batch in one persistent, work-stealing
// launch.  Replaces the reference's host loops over spectra
// (Search.hs:195-201, :232-245) and its per-spectrum b40c sort + full score
// copy-back (Search.hs:250-276).
//
// Planning (all on the device):
//   1. spectra are bucketed by (ion charges, wide/narrow window, 1 Da of
//      precursor residual mass) with a counting sort;
//   2. consecutive spectra of one class form groups of up to G;
//   3. a group's work is the union of its members' candidate windows, cut
//      into chunks of C candidates -- one work item each;
//   4. a persistent grid pulls items from an atomic counter.
// A work item stages its G spectrum rows in shared memory with one bulk
// copy per row (cp.async.bulk + mbarrier), then each warp builds a
// candidate's ion list once and gathers it against every member spectrum
// whose window contains the candidate.  Each warp keeps a register top-K
// per member; the CTA merges them and writes the item's partial lists; a
// merge kernel reduces them per spectrum, and (BF16/FP16 rows) a rescore
// kernel recomputes the kept candidates from the FP32 row.
#include "hfx_internal.h"
#include "device_common.cuh"
#include "batched.h"
#include "batched_common.cuh"
#include "mods_device.cuh"
#include "scan.cuh"
#include "dense.h"
#include <type_traits>

namespace hfx {

constexpr int kMassBuckets = 8192;   // 1 Da buckets of residual mass
constexpr int kClasses = 12;         // (ion charge class 0..5) x (narrow, wide)
constexpr float kWideEps = 1.0f;     // windows wider than this are "wide"

__device__ __forceinline__ int spec_class(const SpecMeta &m) {
    // charge class: plain charges 1..4 (modified ones equal them), 5 = no
    // plain ions but modified ions (charge 6..11), 0 = none
    const int cc = m.charges_plain > 0 ? m.charges_plain : (m.charges_mod > 0 ? 5 : 0);
    return cc * 2 + (m.eps > kWideEps ? 1 : 0);
}
__device__ __forceinline__ int spec_bucket(const SpecMeta &m) {
    int mb = (int)fminf(fmaxf(m.mass, 0.0f), (float)(kMassBuckets - 1));
    return spec_class(m) * kMassBuckets + mb;
}

__global__ void k_bucket_count(const SpecMeta *__restrict__ meta, int32_t nspec, uint32_t *__restrict__ hist) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec) return;
    const SpecMeta m = meta[s];
    if (m.status != 0) return;
    atomicAdd(&hist[spec_bucket(m)], 1u);
}

// Single-CTA exclusive scan of n counters (in place), total in *total.  A warp takes 512 neighbouring counters per round
// in four 16-byte accesses a lane, so the 98,304 mass buckets take six rounds:
// one counter per thread and round took 96, 45 us of a one-spectrum search.
__global__ void __launch_bounds__(1024) k_scan_u32(uint32_t *__restrict__ a, int32_t n, uint32_t *__restrict__ total) {
    __shared__ uint32_t ws[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    const bool wide = on_16(a);
    for (int64_t base = 0; base < n; base += 32 * kScanWarp<uint32_t>) {
        const int64_t at = base + (int64_t)warp * kScanWarp<uint32_t>;
        uint32_t v[kScanSteps][kScanVec<uint32_t>];
        scan_load<uint32_t>(a, n, at, v);
        uint32_t run = 0;
#pragma unroll
        for (int k = 0; k < kScanSteps; ++k) {
            uint32_t own = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) own += v[k][j];
            const uint32_t x = warp_scan_of(own);
            uint32_t e = run + x - own;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t t = v[k][j];
                v[k][j] = e;
                e += t;
            }
            run += __shfl_sync(kFullMask, x, 31);
        }
        if (lane == 0) ws[warp] = run;
        __syncthreads();
        if (warp == 0) ws[lane] = warp_scan_of(ws[lane]);
        __syncthreads();
        const uint32_t before = carry + (warp ? ws[warp - 1] : 0u);
        carry += ws[31];
#pragma unroll
        for (int k = 0; k < kScanSteps; ++k) {
            const int64_t i = at + (int64_t)(k * 32 + lane) * 4;
            if (wide && i + 4 <= n) {
                *reinterpret_cast<uint4 *>(a + i) =
                    make_uint4(before + v[k][0], before + v[k][1], before + v[k][2], before + v[k][3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (i + j < n) a[i + j] = before + v[k][j];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void k_bucket_scatter(const SpecMeta *__restrict__ meta, int32_t nspec, uint32_t *__restrict__ cursor,
                                 int32_t *__restrict__ perm) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec) return;
    const SpecMeta m = meta[s];
    if (m.status != 0) return;
    const uint32_t pos = atomicAdd(&cursor[spec_bucket(m)], 1u);
    perm[pos] = s;
}

// The same for up to kSortFew spectra, by one block without the buckets: a
// spectrum's place is the number of smaller keys (bucket, then number), counted
// over the keys in shared memory.  Of the buckets' ends only the classes' are
// read.  A one-spectrum search took 26 us to clear, count, scan and fill the
// 98,304 buckets; this takes 3 us, and 8 us for 517 spectra, 18 us for 1,024.
__global__ void __launch_bounds__(kSortFew) k_sort_few(const SpecMeta *__restrict__ meta, int32_t nspec,
                                                       uint32_t *__restrict__ bucket_end,
                                                       uint32_t *__restrict__ n_sorted, int32_t *__restrict__ perm) {
    __shared__ __align__(16) uint32_t keys[kSortFew];
    __shared__ uint32_t in_class[kClasses];
    const int t = threadIdx.x;
    uint32_t key = ~0u;  // no row, or no spectrum
    if (t < kClasses) in_class[t] = 0u;
    __syncthreads();
    if (t < nspec) {
        const SpecMeta m = meta[t];
        if (m.status == 0) {
            key = (uint32_t)spec_bucket(m) << 10 | (uint32_t)t;
            atomicAdd(&in_class[spec_class(m)], 1u);
        }
    }
    keys[t] = key;
    __syncthreads();
    if (key != ~0u) {
        uint32_t at = 0;
        for (int j = 0; j < nspec; j += 4) {
            const uint4 k = *reinterpret_cast<const uint4 *>(keys + j);
            at += (k.x < key) + (k.y < key) + (k.z < key) + (k.w < key);
        }
        perm[at] = t;
    }
    if (t < kClasses) {
        uint32_t end = 0;
        for (int c = 0; c <= t; ++c) end += in_class[c];
        bucket_end[(t + 1) * kMassBuckets - 1] = end;
        if (t == kClasses - 1) *n_sorted = end;
    }
}

// With few_groups (no work-item size asked for) a group's window is cut so
// that about kFewItems items come of all groups together, four per resident
// CTA of the list scorer: one spectrum's 3,400 candidates in one item kept one
// SM busy for 0.22 ms.  Groups of narrow and of wide windows count apart; from
// about 1,200 groups (76 of open windows) on the rule changes nothing.
// One thread per group: members, union window, chunk count.
// bucket_end[b] = end of bucket b's spectra in sorted order (the scanned
// counters, which the scatter has moved from the starts to the ends).
__global__ void k_groups(const uint32_t *__restrict__ bucket_end, const uint32_t *__restrict__ n_sorted,
                         const int32_t *__restrict__ perm, const uint32_t *__restrict__ wb,
                         const uint32_t *__restrict__ we, const SpecMeta *__restrict__ meta, int32_t G,
                         int32_t chunk, int few_groups, int32_t max_groups, GroupInfo *__restrict__ groups,
                         uint32_t *__restrict__ nchunks, int32_t *__restrict__ group_of,
                         int32_t *__restrict__ slot_of, uint32_t *__restrict__ ngroups_out) {
    __shared__ uint32_t cls_start[kClasses + 1], grp_start[kClasses + 1];
    if (threadIdx.x == 0) {
        uint32_t gs = 0;
        for (int c = 0; c < kClasses; ++c) {
            cls_start[c] = c ? bucket_end[c * kMassBuckets - 1] : 0u;
            const uint32_t end = bucket_end[(c + 1) * kMassBuckets - 1];
            grp_start[c] = gs;
            gs += (end - cls_start[c] + G - 1) / G;
        }
        cls_start[kClasses] = *n_sorted;
        grp_start[kClasses] = gs;
        if (blockIdx.x == 0) *ngroups_out = gs;
    }
    __syncthreads();
    const int32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= max_groups) return;
    if ((uint32_t)g >= grp_start[kClasses]) {
        nchunks[g] = 0;
        return;
    }
    int c = 0;
    while (c + 1 < kClasses && (uint32_t)g >= grp_start[c + 1]) ++c;
    const uint32_t pos0 = cls_start[c] + ((uint32_t)g - grp_start[c]) * (uint32_t)G;
    const uint32_t cnt = min((uint32_t)G, cls_start[c + 1] - pos0);
    GroupInfo gi;
    gi.pos0 = pos0;
    gi.count = cnt;
    gi.lo = 0xFFFFFFFFu;
    gi.hi = 0u;
    gi.maxlen = 0;
    gi.charges = 0;
    gi.charges_mod = 0;
    gi.block = -1;
    for (uint32_t j = 0; j < cnt; ++j) {
        const int32_t s = perm[pos0 + j];
        group_of[s] = g;
        slot_of[s] = (int32_t)j;
        const uint32_t b = wb[s], e = we[s];
        if (e > b) {
            gi.lo = min(gi.lo, b);
            gi.hi = max(gi.hi, e);
        }
        gi.maxlen = max(gi.maxlen, meta[s].len);
        gi.charges = meta[s].charges_plain;
        gi.charges_mod = meta[s].charges_mod;
    }
    if (gi.hi <= gi.lo) {
        gi.lo = gi.hi = 0;
    }
    // wide windows (open search) are cut into at most ~16 items per group;
    // the groups dispensed last take shorter items (the last quarter 1/4,
    // the last sixteenth 1/16 of the chunk), so the grid ends evenly
    const uint32_t ng = grp_start[kClasses];
    const int32_t cg = (uint32_t)g >= ng - ng / 16 ? max(chunk / 16, 256)
                       : (uint32_t)g >= ng - ng / 4 ? max(chunk / 4, 256)
                                                    : chunk;
    gi.chunk = group_chunk(gi.hi - gi.lo, cg);
    if (few_groups) {
        uint32_t alike = 0;  // groups whose windows are as wide (narrow classes are even, wide ones odd)
        for (int k = c & 1; k < kClasses; k += 2) alike += grp_start[k + 1] - grp_start[k];
        const uint64_t share = ((uint64_t)(gi.hi - gi.lo) * alike + kFewItems - 1) / kFewItems;
        gi.chunk = (uint32_t)min((uint64_t)gi.chunk, max(share, (uint64_t)64));
    }
    groups[g] = gi;
    nchunks[g] = (gi.hi - gi.lo + gi.chunk - 1) / gi.chunk;
}

template <bool FastDiv, typename T, int G>
__global__ void __launch_bounds__(768, 1)
k_score_batched(DevDB db, const T *__restrict__ tiles, int64_t stride, const uint32_t *__restrict__ wb,
                const uint32_t *__restrict__ we, const int32_t *__restrict__ perm,
                const GroupInfo *__restrict__ groups, const uint32_t *__restrict__ item_off,
                const uint32_t *__restrict__ ngroups_p, int32_t chunk, int32_t K, uint32_t *__restrict__ counter,
                float *__restrict__ part_s, uint64_t *__restrict__ part_k, uint32_t *__restrict__ err) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t words_cap = (int32_t)((stride + 31) / 32);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    T *stile = reinterpret_cast<T *>(smem + 128);
    constexpr size_t kQueue = CtaSlots<G>::warp_bytes();
    uint8_t *wbase = smem + 128 + fused_tile_bytes(stride, sizeof(T), G) +
                     (size_t)warp * fused_warp_bytes(words_cap, kQueue);
    uint8_t *my_queue = wbase + fused_queue_offset(words_cap);
    uint32_t *planes = reinterpret_cast<uint32_t *>(wbase);
    uint16_t *list = reinterpret_cast<uint16_t *>(planes + 3 * words_cap);
    __shared__ int32_t s_item;
    __shared__ uint32_t s_next;
    __shared__ uint32_t s_wb[G], s_we[G];
    __shared__ uint32_t thr_u[G], s_lock[G];
    __shared__ float s_ls[G * 32];
    __shared__ uint32_t s_lk[G * 32];

    const int32_t ngroups = (int32_t)*ngroups_p;
    const uint32_t total = item_off[ngroups];
    if (threadIdx.x == 0) mbar_init(bar, 1);
    for (int32_t i = lane; i < 3 * words_cap; i += 32) planes[i] = 0u;
    __syncthreads();
    const Planes pl{planes, planes + words_cap, planes + 2 * words_cap};
    const float mt_lane = db.mt[lane];
    const int my_slot = reduce_slot_of_lane<G>(lane);
    uint32_t phase = 0;
    CtaSlots<G> slots;
    slots.bind(s_ls, s_lk, s_lock, thr_u, my_queue, err);

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
            if (j < cnt_members) {
                const int32_t s = perm[gi.pos0 + j];
                b = wb[s];
                e = we[s];
            }
            s_wb[j] = b;
            s_we[j] = e;
        }
        slots.reset_shared();
        if (threadIdx.x == 0) s_next = p0;
        const int32_t nb = tile_bins(gi.maxlen);
        if (threadIdx.x == 0) {
            fence_proxy_async();
            const uint32_t bytes = (uint32_t)((size_t)nb * G * sizeof(T));
            mbar_arrive_expect_tx(bar, bytes);
            bulk_g2s(stile, tiles + (size_t)g * stride * G, bytes, bar);
        }
        __syncthreads();
        if (!mbar_wait(bar, phase, kWaitLimit)) {
            if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
            return;
        }
        phase ^= 1u;
        const uint32_t my_b = lane < G ? s_wb[lane] : 0u, my_e = lane < G ? s_we[lane] : 0u;
        const TileDot<T, G> dot{stile};
        while (true) {
            // candidates are handed out one at a time so that warps finish together
            uint32_t p = 0;
            if (lane == 0) p = atomicAdd(&s_next, 1u);
            p = __shfl_sync(kFullMask, p, 0);
            if (p >= p1) break;
            const uint32_t act = __ballot_sync(kFullMask, lane < G && my_b <= p && p < my_e) & ((1u << G) - 1u);
            if (!act) continue;
            const WordRange wr = build_planes<FastDiv>(pl, db.ions, db.tc_sorted[p], db.tn_sorted[p],
                                                       db.r_sorted[p], (int)gi.charges, gi.maxlen, mt_lane,
                                                       NoMods{});
            float acc[G];
            planes_accumulate<G>(pl, list, wr, dot, acc);
            const float sc = reduce_scatter<G>(acc);
            const bool want = (lane & (32 / G - 1)) == 0 && ((act >> my_slot) & 1u) &&
                              score_order(sc) >= *(volatile uint32_t *)(thr_u + my_slot);
            slots.offer(want, sc, p, my_slot, K);
        }
        slots.drain(K);
        __syncthreads();  // every warp has merged its queues
        for (int j = warp; j < cnt_members; j += nw) {
            const size_t o = ((size_t)item * G + j) * K;
            slots.result(j, K, part_s + o, part_k + o);
        }
        __syncthreads();
    }
}

// Per spectrum: merge its slot of every item of its group that its window
// reaches, a block of kMergeWarps warps each (one warp over all items of the
// group took 38 us for one spectrum's 53 items, and the windows of a few
// spectra far apart in mass have hundreds).
// R = 1: up to 32 kept per spectrum, R = 2: up to 64.
constexpr int kMergeWarps = 4;
template <int R>
__global__ void __launch_bounds__(32 * kMergeWarps) k_merge_items(const float *__restrict__ part_s, const uint64_t *__restrict__ part_k,
                              const uint32_t *__restrict__ item_off, const int32_t *__restrict__ group_of,
                              const int32_t *__restrict__ slot_of, const SpecMeta *__restrict__ meta,
                              const uint32_t *__restrict__ wb, const uint32_t *__restrict__ we, int32_t G, int32_t K,
                              int32_t kout, float *__restrict__ out_s,
                              uint64_t *__restrict__ out_k, const GroupInfo *__restrict__ groups,
                              const unsigned long long *__restrict__ dense,
                              const unsigned long long *__restrict__ dense_left,
                              const DenseBlock *__restrict__ blocks, const uint32_t *__restrict__ dense_off) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t s = blockIdx.x;
    __shared__ float sm_s[kMergeWarps][32 * R];
    __shared__ uint64_t sm_k[kMergeWarps][32 * R];
    typename std::conditional<R == 1, WarpList32, WarpList64>::type tk;
    tk.init();
    if (meta[s].status == 0) {
        const int32_t g = group_of[s], j = slot_of[s];
        // the items that overlap the spectrum's own window, a warp each in turn
        const GroupInfo gi = groups[g];
        const uint32_t i0 = item_off[g], i1 = item_off[g + 1];
        if (we[s] > wb[s] && i1 > i0) {
            const uint32_t last = min(i1 - 1u, i0 + (we[s] - 1u - gi.lo) / gi.chunk);
            for (uint32_t it = i0 + (wb[s] - gi.lo) / gi.chunk + (uint32_t)warp; it <= last; it += nw) {
                const size_t o = ((size_t)it * G + j) * K;
                tk.merge_list(part_s + o, part_k + o, K);
            }
        }
        // a block scored on the tensor cores: the spectrum's list and what the
        // block's items had left over (unsorted, up to 16 each)
        if constexpr (R == 1) {
            const int32_t b = dense ? gi.block : -1;
            if (b >= 0) {
                auto take = [&](unsigned long long x) {
                    const uint32_t o = (uint32_t)(x >> 32);
                    tk.merge(x ? __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o) : -INFINITY,
                             x ? (uint64_t)(uint32_t)~(uint32_t)x : ~0ull);
                };
                if (warp == 0) take(dense[(size_t)s * 32 + lane]);
                const uint32_t m = gi.pos0 + (uint32_t)j - blocks[b].pos0;
                for (uint32_t it = dense_off[b] + 2u * (uint32_t)warp; it < dense_off[b + 1]; it += 2u * nw) {
                    // two items at a time, 32 entries sorted best first
                    const uint32_t mine = it + (uint32_t)(lane >> 4);
                    unsigned long long x =
                        mine < dense_off[b + 1]
                            ? dense_left[((size_t)mine * kDenseSpectra + m) * kDenseQueue + (lane & 15)]
                            : 0ull;
                    if (!__any_sync(kFullMask, x != 0ull)) continue;
#pragma unroll
                    for (int w = 2; w <= 32; w <<= 1)
#pragma unroll
                        for (int d = w >> 1; d > 0; d >>= 1) {
                            const unsigned long long y = __shfl_xor_sync(kFullMask, x, d);
                            const bool high = ((lane & d) == 0) == ((lane & w) == 0);
                            x = high ? max(x, y) : min(x, y);
                        }
                    take(x);
                }
            }
        }
    }
    // the warps' lists into the first
    if (warp > 0) tk.store(sm_s[warp], sm_k[warp], 32 * R);
    __syncthreads();
    if (warp > 0) return;
    for (int w = 1; w < nw; ++w) tk.merge_list(sm_s[w], sm_k[w], 32 * R);
    tk.store(out_s + (size_t)s * kout, out_k + (size_t)s * kout, kout);
}

// FP32 rescoring of the kept candidates (BF16/FP16-stored rows): one CTA
// per spectrum, each warp recomputes kept entries from the FP32 row, then
// the CTA orders them and writes the top-N.
template <bool FastDiv>
__global__ void __launch_bounds__(256) k_rescore(DevDB db, DevMods mods, const float *__restrict__ rows32,
                                                 int64_t stride, const SpecMeta *__restrict__ meta,
                                                 const float *__restrict__ kept_s,
                                                 const uint64_t *__restrict__ kept_k, int32_t K, int32_t topn,
                                                 float *__restrict__ out_s, uint64_t *__restrict__ out_k,
                                                 uint32_t *__restrict__ out_pep) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t s = blockIdx.x;
    const SpecMeta m = meta[s];
    const int32_t words = (int32_t)((stride + 31) / 32);
    uint32_t *planes = reinterpret_cast<uint32_t *>(smem);
    uint16_t *lists = reinterpret_cast<uint16_t *>(planes + (size_t)nw * 3 * words);
    float *res_s = reinterpret_cast<float *>(lists + (size_t)nw * kListCap);
    uint64_t *res_k = reinterpret_cast<uint64_t *>(res_s + 64);
    for (int32_t i = threadIdx.x; i < nw * 3 * words; i += blockDim.x) planes[i] = 0u;
    __syncthreads();
    Planes pl{planes + (size_t)warp * 3 * words, planes + (size_t)warp * 3 * words + words,
              planes + (size_t)warp * 3 * words + 2 * words};
    uint16_t *list = lists + (size_t)warp * kListCap;
    const float mt_lane = db.mt[lane];
    SpecSet<float, 1> ss;
    ss.row[0] = rows32 + (size_t)s * stride;
    ss.len[0] = m.len;
    ss.active = 1u;
    for (int t = warp; t < K; t += nw) {
        const uint64_t kk = kept_k[(size_t)s * K + t];
        float sc = -INFINITY;
        if (kk != ~0ull && !(kk >> 63)) {
            const uint32_t p = (uint32_t)kk;
            const WordRange wr = build_planes<FastDiv>(pl, db.ions, db.tc_sorted[p], db.tn_sorted[p],
                                                       db.r_sorted[p], m.charges_plain, m.len, mt_lane, NoMods{});
            float acc[1];
            planes_dot<float, 1>(pl, list, wr, ss, acc);
            sc = acc[0];
        } else if (kk != ~0ull) {
            // modified match: combination, mass-order position and isoform rank from the key
            const int32_t mu = (int32_t)((kk >> 54) & 511u);
            const uint32_t p = (uint32_t)((kk >> 27) & ((1u << 27) - 1u));
            const uint32_t rank = (uint32_t)(kk & ((1u << 27) - 1u));
            const uint32_t tc = db.tc_sorted[p], tn = db.tn_sorted[p];
            const int32_t *dcount = mods.counts + (size_t)mu * mods.num_ma;
            uint32_t D[kMaxMa], scan[kMaxMa];
            modable_counts(db.ions, tc, tn, mods.num_ma, D);
            isoform_count(D, dcount, mods.num_ma, scan);
            ModIsoform iso;
            iso.num_ma = mods.num_ma;
            iso.per_type = mods.per_type;
#pragma unroll
            for (int i = 0; i < kMaxMa; ++i) iso.ma_mass[i] = mods.ma_mass[i];
            isoform_masks(D, scan, dcount, mods.num_ma, rank, iso.mask);
            iso.reset();
            const float residual = __fadd_rn(db.r_sorted[p], mods.delta[mu]);
            const WordRange wr = build_planes<FastDiv>(pl, db.ions, tc, tn, residual, m.charges_mod, m.len, mt_lane,
                                                       iso);
            float acc[1];
            planes_dot<float, 1>(pl, list, wr, ss, acc);
            sc = acc[0];
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
            const uint64_t pos = (tk.k >> 63) ? ((tk.k >> 27) & ((1ull << 27) - 1)) : tk.k;
            out_pep[(size_t)s * topn + lane] = (tk.k != ~0ull) ? db.idx_sorted[pos] : ~0u;
        }
    }
}

__global__ void k_finish(const float *__restrict__ in_s, const uint64_t *__restrict__ in_k, int32_t nspec,
                         int32_t topn, const uint32_t *__restrict__ idx_sorted, const uint32_t *__restrict__ wb,
                         const uint32_t *__restrict__ we, const SpecMeta *__restrict__ meta, float *__restrict__ out_s,
                         uint64_t *__restrict__ out_k, uint32_t *__restrict__ out_pep, int32_t plain,
                         const unsigned long long *__restrict__ ncand_mod, int64_t *__restrict__ ncand) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (int64_t)nspec * topn) {
        const uint64_t k = in_k[i];
        out_s[i] = in_s[i];
        out_k[i] = k;
        uint32_t pep = ~0u;
        if (k != ~0ull) {
            const uint64_t pos = (k >> 63) ? ((k >> 27) & ((1ull << 27) - 1)) : k;
            pep = idx_sorted[pos];
        }
        out_pep[i] = pep;
    }
    if (ncand && i < nspec)
        ncand[i] = ((meta[i].status == 0 && plain) ? (int64_t)(we[i] - wb[i]) : 0) +
                   (ncand_mod ? (int64_t)ncand_mod[i] : 0);
}

__global__ void k_ncand(const uint32_t *__restrict__ wb, const uint32_t *__restrict__ we,
                        const SpecMeta *__restrict__ meta, int32_t nspec, int32_t plain,
                        const unsigned long long *__restrict__ ncand_mod, int64_t *__restrict__ ncand) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nspec)
        ncand[i] = ((meta[i].status == 0 && plain) ? (int64_t)(we[i] - wb[i]) : 0) +
                   (ncand_mod ? (int64_t)ncand_mod[i] : 0);
}

}  // namespace hfx

using namespace hfx;

size_t hfx_batched_smem(int64_t stride, int elem_bytes, int G, int nw, int K) {
    (void)K;
    return fused_smem_bytes(stride, elem_bytes, G, nw, cta_queue_bytes(G, 4));
}

int hfx_batched_plan(const SpecMeta *meta, int32_t nspec, const uint32_t *wb, const uint32_t *we, int32_t G,
                     int32_t chunk, int few_groups, const BatchedWs &ws, const DenseWs *dw, cudaStream_t st) {
    const int nbk = kClasses * kMassBuckets;
    cudaMemsetAsync(ws.item_off, 0, sizeof(uint32_t) * (nspec + 1), st);
    if (nspec <= kSortFew) {
        k_sort_few<<<1, kSortFew, 0, st>>>(meta, nspec, ws.hist, ws.n_sorted, ws.perm);
    } else {
        cudaMemsetAsync(ws.hist, 0, sizeof(uint32_t) * (nbk + 1), st);
        k_bucket_count<<<(nspec + 255) / 256, 256, 0, st>>>(meta, nspec, ws.hist);
        k_scan_u32<<<1, 1024, 0, st>>>(ws.hist, nbk, ws.n_sorted);
        k_bucket_scatter<<<(nspec + 255) / 256, 256, 0, st>>>(meta, nspec, ws.hist, ws.perm);
    }
    const int32_t max_groups = nspec;  // each class adds at most one partial group
    k_groups<<<(max_groups + 255) / 256, 256, 0, st>>>(ws.hist, ws.n_sorted, ws.perm, wb, we, meta, G, chunk,
                                                       few_groups, max_groups, ws.groups, ws.item_off, ws.group_of, ws.slot_of,
                                                       ws.ngroups);
    if (dw) {
        const int rc = hfx_dense_plan(meta, nspec, wb, we, G, ws.hist, ws, ws.item_off, *dw, st);
        if (rc) return rc;
        k_scan_u32<<<1, 1024, 0, st>>>(dw->item_off, dw->cap_blocks + 1, dw->total_items);
    }
    k_scan_u32<<<1, 1024, 0, st>>>(ws.item_off, max_groups + 1, ws.total_items);
    return (int)cudaGetLastError();
}

template <bool F, typename T, int G>
static int launch_batched_t(const DevDB &db, const T *rows, int64_t stride, const SpecMeta *meta, const uint32_t *wb,
                            const uint32_t *we, const BatchedWs &ws, void *tiles, uint32_t ngroups, int32_t chunk,
                            int32_t K, int nw, int grid, float *part_s, uint64_t *part_k, uint32_t *err,
                            cudaStream_t st) {
    (void)rows;
    int dev = 0, sms = 0, smem_max = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    auto fn = k_score_batched<F, T, G>;
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, fn);  // static shared memory counts against the same limit
    const size_t avail = (size_t)smem_max > fa.sharedSizeBytes ? (size_t)smem_max - fa.sharedSizeBytes : 0;
    if (nw <= 0) nw = std::min(fused_warps(stride, sizeof(T), G, cta_queue_bytes(G, 4), avail), 24);
    if (nw < 1) return (int)cudaErrorInvalidValue;
    const size_t smem = hfx_batched_smem(stride, sizeof(T), G, nw, K);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    if (grid <= 0) {
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, nw * 32, smem);
        grid = sms * (per > 0 ? per : 1);
    }
    fn<<<grid, nw * 32, smem, st>>>(db, (const T *)tiles, stride, wb, we, ws.perm, ws.groups, ws.item_off,
                                    ws.ngroups, chunk, K, ws.counter, part_s, part_k, err);
    return (int)cudaGetLastError();
}

template <bool F, typename T>
static int launch_batched_g(int G, const DevDB &db, const T *rows, int64_t stride, const SpecMeta *meta,
                            const uint32_t *wb, const uint32_t *we, const BatchedWs &ws, void *tiles, uint32_t ng,
                            int32_t chunk, int32_t K, int nw, int grid, float *ps, uint64_t *pk, uint32_t *err,
                            cudaStream_t st) {
    switch (G) {
    case 1: return launch_batched_t<F, T, 1>(db, rows, stride, meta, wb, we, ws, tiles, ng, chunk, K, nw, grid, ps, pk, err, st);
    case 2: return launch_batched_t<F, T, 2>(db, rows, stride, meta, wb, we, ws, tiles, ng, chunk, K, nw, grid, ps, pk, err, st);
    case 4: return launch_batched_t<F, T, 4>(db, rows, stride, meta, wb, we, ws, tiles, ng, chunk, K, nw, grid, ps, pk, err, st);
    case 8: return launch_batched_t<F, T, 8>(db, rows, stride, meta, wb, we, ws, tiles, ng, chunk, K, nw, grid, ps, pk, err, st);
    default: return (int)cudaErrorInvalidValue;
    }
}

int hfx_batched_score(const DevDB &db, const void *rows, int elem_kind, int64_t stride, const SpecMeta *meta,
                      const uint32_t *wb, const uint32_t *we, const BatchedWs &ws, void *tiles, uint32_t ngroups,
                      int32_t G, int32_t chunk, int32_t K, int nw, int grid, int fastdiv, float *part_s,
                      uint64_t *part_k, uint32_t *err, cudaStream_t st) {
    cudaMemsetAsync(ws.counter, 0, 4, st);
    if (elem_kind == 0) {
        const float *r = (const float *)rows;
        return fastdiv ? launch_batched_g<true, float>(G, db, r, stride, meta, wb, we, ws, tiles, ngroups, chunk, K,
                                                       nw, grid, part_s, part_k, err, st)
                       : launch_batched_g<false, float>(G, db, r, stride, meta, wb, we, ws, tiles, ngroups, chunk, K,
                                                        nw, grid, part_s, part_k, err, st);
    } else if (elem_kind == 1) {
        const __nv_bfloat16 *r = (const __nv_bfloat16 *)rows;
        return fastdiv ? launch_batched_g<true, __nv_bfloat16>(G, db, r, stride, meta, wb, we, ws, tiles, ngroups,
                                                               chunk, K, nw, grid, part_s, part_k, err, st)
                       : launch_batched_g<false, __nv_bfloat16>(G, db, r, stride, meta, wb, we, ws, tiles, ngroups,
                                                                chunk, K, nw, grid, part_s, part_k, err, st);
    } else {
        const __half *r = (const __half *)rows;
        return fastdiv ? launch_batched_g<true, __half>(G, db, r, stride, meta, wb, we, ws, tiles, ngroups, chunk, K,
                                                        nw, grid, part_s, part_k, err, st)
                       : launch_batched_g<false, __half>(G, db, r, stride, meta, wb, we, ws, tiles, ngroups, chunk,
                                                         K, nw, grid, part_s, part_k, err, st);
    }
}

// Graph replays size the work-item buffers from an earlier run: clamp the
// item offsets to that capacity and report an overflow (the host re-plans).
__global__ void k_clamp_items(uint32_t *__restrict__ off, int64_t n1, uint32_t cap, uint32_t *__restrict__ err) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n1) return;
    const uint32_t v = off[i];
    if (v > cap) {
        off[i] = cap;
        if (i == n1 - 1) atomicOr(err, kErrBounds);
    }
}

__global__ void k_clamp_groups(uint32_t *__restrict__ ngroups, uint32_t cap, uint32_t *__restrict__ err) {
    if (threadIdx.x == 0 && *ngroups > cap) {
        *ngroups = cap;
        atomicOr(err, kErrBounds);
    }
}

int hfx_clamp_groups(uint32_t *ngroups, uint32_t cap, uint32_t *err, cudaStream_t st) {
    k_clamp_groups<<<1, 32, 0, st>>>(ngroups, cap, err);
    return (int)cudaGetLastError();
}

int hfx_clamp_items(uint32_t *off, int64_t n1, uint32_t cap, uint32_t *err, cudaStream_t st) {
    if (n1 <= 0) return 0;
    k_clamp_items<<<(unsigned)((n1 + 255) / 256), 256, 0, st>>>(off, n1, cap, err);
    return (int)cudaGetLastError();
}

int hfx_batched_merge(const float *part_s, const uint64_t *part_k, const BatchedWs &ws, const SpecMeta *meta,
                      const uint32_t *wb, const uint32_t *we, int32_t nspec, int32_t G, int32_t K, int32_t kout,
                      float *out_s, uint64_t *out_k,
                      const DenseWs *dw, cudaStream_t st) {
    if (kout > kMaxKept || K > kMaxKept) return (int)cudaErrorInvalidValue;
    if (kout > 32 || K > 32)
        k_merge_items<2><<<nspec, 32 * kMergeWarps, 0, st>>>(part_s, part_k, ws.item_off, ws.group_of, ws.slot_of, meta,
                                                          wb, we, G, K, kout, out_s, out_k, ws.groups,
                                                          dw ? dw->best : nullptr, dw ? dw->left : nullptr,
                                                          dw ? dw->blocks : nullptr, dw ? dw->item_off : nullptr);
    else
        k_merge_items<1><<<nspec, 32 * kMergeWarps, 0, st>>>(part_s, part_k, ws.item_off, ws.group_of, ws.slot_of, meta,
                                                          wb, we, G, K, kout, out_s, out_k, ws.groups,
                                                          dw ? dw->best : nullptr, dw ? dw->left : nullptr,
                                                          dw ? dw->blocks : nullptr, dw ? dw->item_off : nullptr);
    return (int)cudaGetLastError();
}

int hfx_rescore(const DevDB &db, const DevMods &mods, const float *rows32, int64_t stride, const SpecMeta *meta,
                const float *kept_s,
                const uint64_t *kept_k, int32_t nspec, int32_t K, int32_t topn, int fastdiv, float *out_s,
                uint64_t *out_k, uint32_t *out_pep, cudaStream_t st) {
    const int nw = 8;
    const int32_t words = (int32_t)((stride + 31) / 32);
    const size_t smem = (size_t)nw * 3 * words * 4 + (size_t)nw * kListCap * 2 + 64 * 4 + 64 * 8;
    auto f = fastdiv ? k_rescore<true> : k_rescore<false>;
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    f<<<nspec, nw * 32, smem, st>>>(db, mods, rows32, stride, meta, kept_s, kept_k, K, topn, out_s, out_k, out_pep);
    return (int)cudaGetLastError();
}

int hfx_finish(const float *in_s, const uint64_t *in_k, int32_t nspec, int32_t topn, const uint32_t *idx_sorted,
               const uint32_t *wb, const uint32_t *we, const SpecMeta *meta, float *out_s, uint64_t *out_k,
               uint32_t *out_pep, int32_t plain, const unsigned long long *ncand_mod, int64_t *ncand,
               cudaStream_t st) {
    const int64_t n = std::max<int64_t>((int64_t)nspec * topn, nspec);
    k_finish<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in_s, in_k, nspec, topn, idx_sorted, wb, we, meta, out_s,
                                                          out_k, out_pep, plain, ncand_mod, ncand);
    return (int)cudaGetLastError();
}

int hfx_ncand(const uint32_t *wb, const uint32_t *we, const SpecMeta *meta, int32_t nspec, int32_t plain,
              const unsigned long long *ncand_mod, int64_t *ncand, cudaStream_t st) {
    k_ncand<<<(nspec + 255) / 256, 256, 0, st>>>(wb, we, meta, nspec, plain, ncand_mod, ncand);
    return (int)cudaGetLastError();
}

template <typename T>
static int pack_tiles_g(int32_t G, const void *rows, int64_t stride, const SpecMeta *meta, const BatchedWs &ws,
                        void *tiles, uint32_t ngroups, cudaStream_t st) {
    if (ngroups == 0) return 0;
    const T *r = (const T *)rows;
    if (G == 16) hfx_pack_tiles_launch<T, 16>(r, stride, meta, ws, (T *)tiles, ngroups, st);
    else if (G == 8) hfx_pack_tiles_launch<T, 8>(r, stride, meta, ws, (T *)tiles, ngroups, st);
    else if (G == 4) hfx_pack_tiles_launch<T, 4>(r, stride, meta, ws, (T *)tiles, ngroups, st);
    else if (G == 2) hfx_pack_tiles_launch<T, 2>(r, stride, meta, ws, (T *)tiles, ngroups, st);
    else if (G == 1) hfx_pack_tiles_launch<T, 1>(r, stride, meta, ws, (T *)tiles, ngroups, st);
    else return (int)cudaErrorInvalidValue;
    return (int)cudaGetLastError();
}

int hfx_pack_tiles(const void *rows, int elem_kind, int64_t stride, const SpecMeta *meta, const BatchedWs &ws,
                   void *tiles, uint32_t ngroups, int32_t G, cudaStream_t st) {
    if (elem_kind == 0) return pack_tiles_g<float>(G, rows, stride, meta, ws, tiles, ngroups, st);
    if (elem_kind == 1) return pack_tiles_g<__nv_bfloat16>(G, rows, stride, meta, ws, tiles, ngroups, st);
    return pack_tiles_g<__half>(G, rows, stride, meta, ws, tiles, ngroups, st);
}
