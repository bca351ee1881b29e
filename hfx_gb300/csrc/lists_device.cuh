// Device helpers of the per-step ion lists, shared by the list kernels of
// unmodified candidates (lists.cu) and of modified isoforms (iso_lists.cu).
#pragma once
#include <cstdint>
#include "device_common.cuh"

namespace hfx {

// The ascending distinct-bin lists of one candidate, level by level.
//
// One warp holds one candidate.  A list entry's place is the number of
// distinct bins below it, so no sort and no walk over the set bits is needed:
// the warp marks the charge-z bins in a bit per bin, one scan over the words
// gives each word the number of set bits before it, and every lane then looks
// up the place of its own ions' bins (prefix + popcount below the bit) and
// writes their entries there.  The level-(z-1) list, whose bins are a subset,
// is carried over by the same lookup, 32 entries at a time.  An entry's level
// is the highest of its ions (ion_series.cu:71-75 atomicMax): levels are
// written in ascending order (neutral losses and a-ions, the previous list,
// the flanks where no 50 stands, the 50s), so nothing is looked up to find it.
//
// What bounds it: instruction issue and shared-memory wavefronts.  Against
// three bit planes compacted by a bit loop per lane (up to 16 of 32 lanes
// active, ~990 warp instructions a list) this takes about a third of the
// instructions; the figures are at k_gen_lists and k_gen_iso_lists.
//
// Shared memory is addressed by 32-bit shared addresses: a pointer that could
// be generic made every access pay for it (and the atomics above all).
struct RankBufs {
    uint32_t pl;      // words of (a bit per bin, set bits before the word), 8 bytes each
    uint32_t a, b;    // the level's list and the previous one, kStageCap 16-bit entries each
    int32_t words;    // a multiple of 2
};

// Room of one staged list of a warp (entries): lists up to this long are
// built in shared memory and copied out in 16-byte pieces; a candidate with a
// longer one is left to a second kernel that builds it in global memory
// (build_lists_direct: a call from the staged kernel took its registers from
// 56 to 127).
constexpr int kStageCap = 1024;

// Bin x has bit x + 2, so that an ion's neighbours and bins outside the row
// have bits of their own (0, 1 and nbins + 2 .. nbins + 4) and marking needs no
// test; rank_scan drops those.
__host__ __device__ __forceinline__ int32_t rank_words(int32_t nbins) { return (((nbins + 2) >> 5) + 3) & ~1; }
// Lanes that hold a candidate of a class, and its staging room: a ladder of up
// to 16 prefixes takes half a warp.  The generators are bound by instructions
// issued per warp, and the mean ladder has 16 prefixes: one candidate a warp
// left half its lanes idle.
__host__ __device__ constexpr int class_lanes(int cls) { return cls == 3 ? 16 : 32; }
__host__ __device__ constexpr int class_cap(int cls) { return cls == 3 ? 640 : kStageCap; }  // 640 = 16 prefixes x 4 charges x 10
// Shared memory of one candidate (a multiple of 16 bytes).
__host__ __device__ __forceinline__ size_t rank_bytes(int32_t nbins, int cls) {
    return (size_t)rank_words(nbins) * 8 + (size_t)2 * class_cap(cls) * 2;
}
__device__ __forceinline__ RankBufs rank_bufs(const uint8_t *base, int32_t nbins, int cls) {
    RankBufs rb;
    rb.words = rank_words(nbins);
    rb.pl = smem_u32(base);
    rb.a = rb.pl + (uint32_t)rb.words * 8u;
    rb.b = rb.a + (uint32_t)class_cap(cls) * 2u;
    return rb;
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint2 lds_u64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 lds_u128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(a)
                 : "memory");
    return v;
}
__device__ __forceinline__ void sts_u16(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add(uint32_t a, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t atom_add(uint32_t a, uint32_t v) {
    uint32_t o;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ void sts_u128(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}
// The same under a predicate x < limit (unsigned), without a branch.
__device__ __forceinline__ void sts_u16_lt(uint32_t a, uint32_t v, uint32_t x, uint32_t limit) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %2, %3;\n\t@p st.shared.u16 [%0], %1;\n\t}" ::"r"(a),
                 "h"((uint16_t)v), "r"(x), "r"(limit)
                 : "memory");
}
__device__ __forceinline__ uint32_t lds_u16_lt(uint32_t a, uint32_t x, uint32_t limit, uint32_t otherwise) {
    uint32_t v;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u16 h;\n\tsetp.lt.u32 p, %2, %3;\n\tcvt.u16.u32 h, %4;\n\t"
        "@p ld.shared.u16 h, [%1];\n\tcvt.u32.u16 %0, h;\n\t}"
        : "=r"(v)
        : "r"(a), "r"(x), "r"(limit), "r"(otherwise)
        : "memory");
    return v;
}
__device__ __forceinline__ void red_or_lt(uint32_t a, uint32_t v, uint32_t x, uint32_t limit) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %2, %3;\n\t@p red.shared.or.b32 [%0], %1;\n\t}" ::"r"(a),
                 "r"(v), "r"(x), "r"(limit)
                 : "memory");
}

// Where a candidate's lists go: the level-z list at base + a z(z-1)/2 + b z,
// its length at len[(z - 1) len_step].
struct ListSlots {
    uint16_t *base;
    uint64_t a, b;
    uint16_t *len;
    uint64_t len_step;
    __device__ __forceinline__ uint16_t *slot(int z) const {
        return base + a * (uint64_t)(z * (z - 1) / 2) + b * (uint64_t)z;
    }
};

// The b-ladder of residues [base, base + cnt), cnt <= W, after `carry`: the
// reference warp scan (ion_series.cu:25-56, 176-213), lane i of the W prefix i
// (for 16 its last stride moves nothing).
template <int W = 32, typename Mods>
__device__ __forceinline__ float ladder_chunk(const uint8_t *__restrict__ ions, uint32_t base, int cnt,
                                              float mt_lane, Mods &mods, float carry) {
    const int lane = threadIdx.x & (W - 1);
    uint32_t byte = 0;
    if (lane < cnt) byte = __ldg(ions + base + lane);
    float v = residue_mass(mt_lane, byte);
    const float add = mods.chunk_add(byte, lane < cnt, lane);
    if (add != 0.0f) v = __fadd_rn(v, add);
    if (lane >= cnt) v = 0.0f;
    if (lane == 0) v = __fadd_rn(v, carry);
#pragma unroll
    for (int d = 1; d < W; d <<= 1) {
        const float t = __shfl_up_sync(kFullMask, v, d, W);
        if (lane >= d) v = __fadd_rn(v, t);
    }
    return v;
}

// The bits of one (prefix, charge)'s ions: the a-ion, the b-ion's water and
// ammonia losses and the y-ion's ammonia loss (10 each), and the first of the
// three bits of the b- and of the y-ion (25, 50, 25; ion_series.cu:78-123).
// A bin past the row's end gets bit nbins + 2, past the row's bits; x = -1, the
// conversion's largest value, keeps its neighbour 0 as in 32-bit arithmetic.
struct ItemBits {
    uint32_t s[4], t[2];
};

// Correctly rounded a / d from y = RN(1 / d): q = RN(a y) is within an ulp, the
// remainder a - q d is exact in one FMA, and q + remainder y rounds to the
// quotient (Markstein, IBM J. Res. Dev. 34, 1990).  Equal to the IEEE division
// for d = 1.0005079, 0.02 and 3 and every float in [2^-12, 2^22], which is where
// the ions lie (all of them compared once with the division;
// tests/test_lists_math.py compares some of them in exact arithmetic.  An
// infinite a would give a NaN, so masses from 2^22 on take the other path).  Three instructions and no branch;
// the division's own slow path is a call, which costs a kernel that keeps a
// candidate in registers 16 of them and spills.
__device__ __forceinline__ float quotient(float a, float d, float y) {
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-q, d, a), y, q);
}

// kSmall: every mass is below 2^22 (quotient), else the general division.
template <bool FastDiv, bool kSmall>
__device__ __forceinline__ uint32_t ion_bin(float mz) {
    if constexpr (FastDiv || !kSmall) return (uint32_t)bin_of<FastDiv>(mz);
    else return __float2uint_rz(rintf(quotient(mz, kBinMono, kInvBinMono)));
}
// rz = RN(1 / z): one form for every charge (exact scalings for 1, 2 and 4), no branch.
template <bool FastDiv, bool kSmall>
__device__ __forceinline__ float ion_mz(float a, int z, float rz) {
    if constexpr (FastDiv || !kSmall) return div_charge<FastDiv>(a, z);
    else return quotient(a, (float)z, rz);
}

template <bool FastDiv, bool kSmall>
__device__ __forceinline__ ItemBits item_bits(float b, float y, const ChargeConst &k, float rz, uint32_t nbins) {
    auto single = [&](float mz) { return min(ion_bin<FastDiv, kSmall>(mz) + 2u, nbins + 2u); };
    auto triple = [&](float mz) { return min(ion_bin<FastDiv, kSmall>(mz) + 1u, nbins + 2u); };
    ItemBits t;
    t.s[0] = single(ion_mz<FastDiv, kSmall>(__fadd_rn(__fsub_rn(b, kCO), k.hc), k.c, rz));
    float m = ion_mz<FastDiv, kSmall>(__fadd_rn(b, k.hc), k.c, rz);
    t.t[0] = triple(m);
    t.s[1] = single(__fsub_rn(m, k.dh2o));
    t.s[2] = single(__fsub_rn(m, k.dnh3));
    m = ion_mz<FastDiv, kSmall>(__fadd_rn(__fadd_rn(y, kH2O), k.hc), k.c, rz);
    t.t[1] = triple(m);
    t.s[3] = single(__fsub_rn(m, k.dnh3));
    return t;
}

__device__ __forceinline__ uint32_t word_addr(uint32_t pl, uint32_t bit) { return pl + ((bit >> 5) << 3); }

__device__ __forceinline__ void mark_item(uint32_t pl, const ItemBits &t, uint32_t nbins) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
        red_or_lt(word_addr(pl, t.s[k]), __funnelshift_l(0u, 1u, t.s[k]), t.s[k] - 2u, nbins);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t w = word_addr(pl, t.t[k]);
        red_or_lt(w, __funnelshift_l(0u, 7u, t.t[k]), t.t[k], nbins + 2u);
        // the bits beyond the word, when the first is its bit 30 or 31
        red_or_lt(w + 8u, __funnelshift_l(7u, 0u, t.t[k]), 29u, t.t[k] < nbins + 2u ? t.t[k] & 31u : 0u);
    }
}

// Drops the bits outside the row, then the set bits before each of the first
// `words` words; returns the number of set bits.  A lane takes two
// neighbouring words, 16 bytes: free of bank conflicts (four words a lane in
// two accesses took eight wavefronts each, 40 % of the kernel's).
template <int W = 32>
__device__ __forceinline__ int rank_scan(uint32_t pl, int32_t words, uint32_t nbins) {
    const int lane = threadIdx.x & (W - 1);
    if (lane < 3) {
        const uint32_t top = nbins + 2u;
        const uint32_t at = lane == 0 ? pl : word_addr(pl, top) + (lane == 2 ? 8u : 0u);
        const uint32_t keep = lane == 0 ? ~3u : (lane == 1 ? (1u << (top & 31u)) - 1u : 0u);
        asm volatile("red.shared.and.b32 [%0], %1;" ::"r"(at), "r"(keep) : "memory");
    }
    __syncwarp();
    int before = 0;
#pragma unroll 1
    for (int w0 = 0; w0 < words; w0 += 2 * W) {
        const int w = w0 + 2 * lane;
        const uint32_t at = pl + 8u * (uint32_t)w;
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
        if (w < words) u = lds_u128(at);
        const int c0 = __popc(u.x), c1 = c0 + __popc(u.z);
        int incl = c1;
#pragma unroll
        for (int d = 1; d < W; d <<= 1) {
            const int t = __shfl_up_sync(kFullMask, incl, d, W);
            if (lane >= d) incl += t;
        }
        u.y = (uint32_t)(before + incl - c1);
        u.w = u.y + (uint32_t)c0;
        if (w < words) sts_u128(at, u);
        before += __shfl_sync(kFullMask, incl, W - 1, W);
    }
    __syncwarp();
    return before;
}

// The set bits below `bit`: its place in the list.
__device__ __forceinline__ uint32_t rank_in(uint2 e, uint32_t bit) {
    return e.y + (uint32_t)__popc(e.x & ~__funnelshift_l(0u, ~0u, bit));
}
__device__ __forceinline__ uint32_t rank_of(uint32_t pl, uint32_t bit) { return rank_in(lds_u64(word_addr(pl, bit)), bit); }

// The level lists of one candidate with up to W NC prefixes (NC = 1 or 2), held
// by W lanes (two candidates a warp for 16: the warp-wide steps are common to
// both, and the levels go up to the higher one's), its ladder and the level's
// bins kept in registers between marking and placing.  `need`: bit z - 1 asks for the level-z list.  Returns the entries
// written, or -1 when a list does not fit the staging buffers (or a mass is
// out of `quotient`'s range).  The bits are left cleared.
template <bool FastDiv, int NC, int W, typename Mods>
__device__ __forceinline__ int build_lists_staged(const RankBufs &rb, const uint8_t *__restrict__ ions, uint32_t tc,
                                                  int len, float residual, uint32_t need, uint32_t nbins,
                                                  float mt_lane, Mods mods, const ListSlots &ls) {
    const int lane = threadIdx.x & (W - 1);
    const int zmax = 32 - __clz(__reduce_or_sync(kFullMask, need));  // of the warp's candidates
    const uint32_t pl = rb.pl;
    float v[NC], y[NC];
    float carry = 0.0f, top = 0.0f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        v[c] = ladder_chunk<W>(ions, tc + (uint32_t)(W * c), min(W, len - W * c), mt_lane, mods, carry);
        if (c + 1 < NC) carry = __shfl_sync(kFullMask, v[c], W - 1, W);
        y[c] = __fsub_rn(residual, v[c]);
        // lanes past the end: ions past every row, which nothing below marks or writes
        if (lane + W * c < len) top = fmaxf(top, fmaxf(v[c], y[c]));
        else v[c] = y[c] = 0x1p21f;
    }
    // no ion lies above its prefix or suffix mass + H2O + H: the words in use
    const uint32_t hi = __reduce_max_sync(kFullMask, __float2uint_rz(__fadd_rn(top, 24.0f)));
    if (hi >= (1u << 21)) return -1;  // (either candidate's: both are left)
    const int32_t words = rank_words((int32_t)min(hi, nbins));
    uint32_t dst = rb.a, prev = rb.b;
    int n_prev = 0, entries = 0;
#pragma unroll 1
    for (int z = 1; z <= zmax; ++z) {
        ChargeConst kc;
        kc.c = z;
        kc.hc = __fmul_rn(kH, (float)z);
        const float rz = z == 1 ? 1.0f : (z == 2 ? 0.5f : (z == 3 ? 1.0f / 3.0f : 0.25f));
        kc.dh2o = ion_mz<FastDiv, true>(kH2O, z, rz);
        kc.dnh3 = ion_mz<FastDiv, true>(kNH3, z, rz);
        ItemBits t[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            t[c] = item_bits<FastDiv, true>(v[c], y[c], kc, rz, nbins);
            mark_item(pl, t[c], nbins);
        }
        __syncwarp();
        const int n = rank_scan<W>(pl, words, nbins);
        if (W == 32 && n > kStageCap) {  // (16 prefixes' lists always fit)
            entries = -1;
            break;
        }
        // entries that are not carried over read as no level
#pragma unroll 1
        for (int i = lane; i < ((n + 7) >> 3); i += W) sts_u128(dst + 16u * i, make_uint4(0u, 0u, 0u, 0u));
        __syncwarp();
        // level 1 (10); bit s is bin s - 2
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            uint2 e[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) e[k] = lds_u64(word_addr(pl, t[c].s[k]));
#pragma unroll
            for (int k = 0; k < 4; ++k)
                sts_u16_lt(dst + 2u * rank_in(e[k], t[c].s[k]), t[c].s[k] * 4u - 7u, t[c].s[k] - 2u, nbins);
        }
        __syncwarp();
        // the previous level's list at its new places, two entries a lane
#pragma unroll 1
        for (int i = 2 * lane; i < n_prev; i += 2 * W) {
            const uint32_t p = lds_u32(prev + 2u * i);
            const uint32_t s0 = ((p & 0xFFFFu) >> 2) + 2u, s1 = i + 1 < n_prev ? (p >> 18) + 2u : 0u;
            const uint2 e0 = lds_u64(word_addr(pl, s0)), e1 = lds_u64(word_addr(pl, s1));
            sts_u16(dst + 2u * rank_in(e0, s0), p);
            sts_u16_lt(dst + 2u * rank_in(e1, s1), p >> 16, s1 - 1u, ~0u);
        }
        __syncwarp();
        // level 2 (25) beside each 50, where the carried-over list holds no
        // 50; the three bins' places follow one another
        uint32_t centre[NC][2];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            uint32_t r[2], f[4];
#pragma unroll
            for (int k = 0; k < 2; ++k) r[k] = dst + 2u * rank_of(pl, t[c].t[k]);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t b = t[c].t[k];
                centre[c][k] = r[k] + (b - 2u < nbins ? 2u : 0u);
                f[2 * k] = lds_u16_lt(r[k], b - 2u, nbins, 3u);
                f[2 * k + 1] = lds_u16_lt(centre[c][k] + (b - 1u < nbins ? 2u : 0u), b, nbins, 3u);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t b = t[c].t[k];
                sts_u16_lt(r[k], b * 4u - 6u, f[2 * k] & 3u, 3u);
                sts_u16_lt(centre[c][k] + (b - 1u < nbins ? 2u : 0u), b * 4u + 2u, f[2 * k + 1] & 3u, 3u);
            }
        }
        __syncwarp();
        // level 3 (50)
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int k = 0; k < 2; ++k) sts_u16_lt(centre[c][k], t[c].t[k] * 4u - 1u, t[c].t[k] - 1u, nbins);
        __syncwarp();
        if ((need >> (z - 1)) & 1u) {
            // 16-byte copies: slot and staged list start on 16-byte
            // boundaries and hold n rounded up to 8 entries
            uint4 *out = reinterpret_cast<uint4 *>(ls.slot(z));
#pragma unroll 1
            for (int i = lane; i < ((n + 7) >> 3); i += W) out[i] = lds_u128(dst + 16u * i);
            if (lane == 0) ls.len[(uint64_t)(z - 1) * ls.len_step] = (uint16_t)n;
            entries += n;
        }
        n_prev = n;
        const uint32_t swap = dst;
        dst = prev;
        prev = swap;
    }
#pragma unroll 1
    for (int i = lane; i < (words >> 1); i += W) sts_u128(pl + 16u * i, make_uint4(0u, 0u, 0u, 0u));
    __syncwarp();
    return entries;
}

// The same for a candidate of any length whose lists may outgrow the staging
// buffers: the lists are built in their slots in global memory (every level
// up to the highest needed has one), the ladder and the bins once per pass.
template <bool FastDiv, typename Mods>
__device__ __forceinline__ int build_lists_direct(const RankBufs &rb, const uint8_t *__restrict__ ions, uint32_t tc,
                                                  int len, float residual, uint32_t need, uint32_t nbins,
                                                  float mt_lane, const Mods &mods, const ListSlots &ls) {
    const int lane = threadIdx.x & 31;
    const int zmax = 32 - __clz(need);
    const uint32_t pl = rb.pl;
    int n_prev = 0, entries = 0;
    for (int z = 1; z <= zmax; ++z) {
        const ChargeConst kc = charge_const<FastDiv>(z);
        uint16_t *dst = ls.slot(z);
        int n = 0;
        // pass 0 marks, then 1 (10), the previous list, 2 (25) and 3 (50)
        for (int pass = 0; pass < 4; ++pass) {
            if (pass == 1) {
                n = rank_scan(pl, rb.words, nbins);
#pragma unroll 1
                for (int i = lane; i < n; i += 32) dst[i] = 0;
                __syncwarp();
            }
            if (pass == 2 && z > 1) {
                const uint16_t *prev = ls.slot(z - 1);
#pragma unroll 1
                for (int i = lane; i < n_prev; i += 32) {
                    const uint32_t e = prev[i];
                    dst[rank_of(pl, (e >> 2) + 2u)] = (uint16_t)e;
                }
                __syncwarp();
            }
            float carry = 0.0f;
            Mods m = mods;
            for (int k0 = 0; k0 < len; k0 += 32) {
                const int cnt = min(32, len - k0);
                const float v = ladder_chunk(ions, tc + (uint32_t)k0, cnt, mt_lane, m, carry);
                carry = __shfl_sync(kFullMask, v, cnt - 1);
                if (lane < cnt) {
                    const ItemBits t = item_bits<FastDiv, false>(v, __fsub_rn(residual, v), kc, 0.0f, nbins);
                    auto put = [&](uint32_t bit, uint32_t lvl) {
                        if (bit - 2u < nbins) {
                            uint16_t *at = dst + rank_of(pl, bit);
                            if ((*at & 3u) < lvl) *at = (uint16_t)(bit * 4u - 8u + lvl);
                        }
                    };
                    if (pass == 0) mark_item(pl, t, nbins);
                    for (int k = 0; k < 4 && pass == 1; ++k) put(t.s[k], 1u);
                    for (int k = 0; k < 2 && pass == 2; ++k) {
                        put(t.t[k], 2u);
                        put(t.t[k] + 2u, 2u);
                    }
                    for (int k = 0; k < 2 && pass == 3; ++k) put(t.t[k] + 1u, 3u);
                }
                __syncwarp();
            }
            __syncwarp();
        }
        if ((need >> (z - 1)) & 1u) {
            if (lane == 0) ls.len[(uint64_t)(z - 1) * ls.len_step] = (uint16_t)n;
            entries += n;
        }
        n_prev = n;
    }
#pragma unroll 1
    for (int i = lane; i < (rb.words >> 1); i += 32) sts_u128(pl + 16u * i, make_uint4(0u, 0u, 0u, 0u));
    __syncwarp();
    return entries;
}

// The kernel a candidate's lists are built by: class 3 holds ladders of up to 16
// prefixes, two a warp, class 1 and 2 ladders of up to 32 and 64 (kept apart
// because two chunks cost every candidate spills), class 0 is the rest
// (build_lists_direct).
__device__ __forceinline__ int list_class(uint32_t tc, uint32_t tn) {
    const uint32_t len = tn > tc ? tn - tc : 0u;
    return len <= 16u ? 3 : (len <= 32u ? 1 : (len <= 64u ? 2 : 0));
}

// Work lists of the four classes: counts at w[0..3], then `cap` entries each.
struct WorkLists {
    uint32_t *w;
    uint64_t cap;
    __device__ __forceinline__ uint32_t count(int c) const { return w[c]; }
    __device__ __forceinline__ uint32_t *list(int c) const { return w + 4 + (uint64_t)c * cap; }
};
constexpr int kWorkLists = 4;
__host__ __device__ __forceinline__ size_t work_words(uint64_t cap) { return 4 + kWorkLists * (size_t)cap; }

// Appends `value` to list `cls` (none when negative); every thread of the
// block calls it.  One global atomic per block and class.
__device__ __forceinline__ void append_work(const WorkLists &wl, int cls, uint32_t value) {
    __shared__ uint32_t s_n[kWorkLists], s_base[kWorkLists];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < kWorkLists) s_n[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t at = 0;
#pragma unroll
    for (int c = 0; c < kWorkLists; ++c) {
        const uint32_t bal = __ballot_sync(kFullMask, cls == c);
        uint32_t base = 0;
        if (lane == 0 && bal) base = atomicAdd(&s_n[c], (uint32_t)__popc(bal));
        base = __shfl_sync(kFullMask, base, 0);
        if (cls == c) at = base + (uint32_t)__popc(bal & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (threadIdx.x < kWorkLists && s_n[threadIdx.x]) s_base[threadIdx.x] = atomicAdd(wl.w + threadIdx.x, s_n[threadIdx.x]);
    __syncthreads();
    if (cls >= 0) wl.list(cls)[s_base[cls] + at] = value;
}

// All needed level lists of one candidate of the class: the entries written, or
// -1 when it is one for class 0 after all.
template <bool FastDiv, int kClass, typename Mods>
__device__ __forceinline__ int build_lists(const RankBufs &rb, const uint8_t *__restrict__ ions, uint32_t tc,
                                           uint32_t tn, float residual, uint32_t need, uint32_t nbins, float mt_lane,
                                           const Mods &mods, const ListSlots &ls) {
    const int len = tn > tc ? (int)(tn - tc) : 0;
    if constexpr (kClass == 0)
        return build_lists_direct<FastDiv>(rb, ions, tc, len, residual, need, nbins, mt_lane, mods, ls);
    else
        return build_lists_staged<FastDiv, kClass == 2 ? 2 : 1, class_lanes(kClass)>(rb, ions, tc, len, residual, need,
                                                                                    nbins, mt_lane, mods, ls);
}

// A lane's entries of one round over a list of n, W lanes to a list: entry k of
// the round's 4 W is lane k % W's, the canonical order of FP32 sums.  BF16/FP16
// sums may take any order, but neighbouring entries (an ion's three bins) then
// meet in one access: with four or eight of them a lane, in one load of 8 or 16
// bytes, the scorers were slower (2.90 against 2.74 ms, 65 against 55 ms at
// 0.02 Da, isoforms 15.0 against 14.0 ms).
template <typename E, int W>
struct EntryRound {
    static constexpr int kRound = 4 * W;
    uint32_t e[4];
    __device__ __forceinline__ void load(const E *lp, int i0, int hl, int n, uint32_t pad) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + W * k + hl;
            e[k] = i < n ? (uint32_t)__ldg(lp + i) : pad;
        }
    }
};

// Offset of the list of (level z, mass-order position p): every level has a
// static region; position p's slot holds z * (10 (tn - tc) rounded up to 8)
// entries and starts on a 16-byte boundary.
__device__ __forceinline__ uint64_t list_offset(const uint32_t *__restrict__ lstart, uint64_t total10, int z,
                                                uint32_t p) {
    return total10 * (uint64_t)(z * (z - 1) / 2) + (uint64_t)z * lstart[p];
}

}  // namespace hfx
