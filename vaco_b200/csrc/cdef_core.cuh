// cdef_core.cuh -- CDEF device functions shared by the CDEF kernels and the
// fused deblock+CDEF kernel.  Mirrors vaco crates/codec/vaco-codec-av1/src/cdef.rs
// (find_direction :79, constrain :126, filter_block :142, adjust_strength
// :209, chroma_direction :224).
//
// Unavailable neighbours (outside the plane, apply_cdef's availability rule,
// src/decode.rs:828-831) are stored as the sentinel kSent: constrain() of a
// sentinel difference is 0 for every valid strength/damping pair and the
// maximum masks it out with kMaxMask, so no tap needs a bounds check.
#pragma once

#include "common.cuh"

namespace vaco {
namespace cdefk {

constexpr int kSent = 0xC000;      // > any 12-bit sample; & kMaxMask == 0
constexpr int kMaxMask = 0x3FFF;

// (row, col) step per direction and distance (src/cdef.rs:57-66).
struct DirTable {
    int8_t v[8][2][2];
};
constexpr DirTable kDir = {{
    {{-1, 1}, {-2, 2}}, {{0, 1}, {-1, 2}}, {{0, 1}, {0, 2}},  {{0, 1}, {1, 2}},
    {{1, 1}, {2, 2}},   {{1, 0}, {2, 1}},  {{1, 0}, {2, 0}},  {{1, 0}, {2, -1}},
}};
// The table packed into one 24-bit immediate per (distance, axis): 3 bits
// per direction, biased by 2.  A lookup with a per-lane direction is then a
// shift and a mask instead of a divergent constant-memory read.
__host__ __device__ constexpr uint32_t dir_packed(int k, int axis) {
    uint32_t m = 0;
    for (int d = 0; d < 8; ++d) m |= (uint32_t)(kDir.v[d][k][axis] + 2) << (3 * d);
    return m;
}
template <int K, int AXIS>
__device__ __forceinline__ int dir_step(int d) {
    constexpr uint32_t m = dir_packed(K, AXIS);
    return (int)((m >> (3 * d)) & 7u) - 2;
}
// Sample offset of tap distance K along direction d in a plane of `pitch`.
template <int K>
__device__ __forceinline__ int dir_offset(int d, int pitch) {
    return dir_step<K, 0>(d) * pitch + dir_step<K, 1>(d);
}

// Line index of pixel (i, j) for direction d (src/cdef.rs:88-97).
__host__ __device__ constexpr int dir_bin(int d, int i, int j) {
    return d == 0 ? i + j : d == 1 ? i + j / 2 : d == 2 ? i : d == 3 ? 3 + i - j / 2
         : d == 4 ? 7 + i - j : d == 5 ? 3 + j - i / 2 : d == 6 ? j : i / 2 + j;
}
__host__ __device__ constexpr int dir_count(int d, int b) {
    int n = 0;
    for (int i = 0; i < 8; ++i)
        for (int j = 0; j < 8; ++j) n += dir_bin(d, i, j) == b;
    return n;
}
__host__ __device__ constexpr int dir_weight(int d, int b) {
    return dir_count(d, b) ? 840 / dir_count(d, b) : 0;
}

// How a direction's lines meet the words of two samples that a row is read as
// (word k of row i: samples 2k, 2k+1).
constexpr bool dir_word_in_one_line(int d) { return dir_bin(d, 0, 0) == dir_bin(d, 0, 1); }  // 1, 2, 3
constexpr bool dir_row_pair(int d) { return dir_bin(d, 0, 0) == dir_bin(d, 1, 0); }          // 5, 6, 7

// Sum over the lines of direction D of (line sum)^2 * 840 / (line length) for
// the 8-bit samples of a block, two per word in w[row][word].
//
// vaco subtracts 128 from every sample first (src/cdef.rs:99-112).  With 840 /
// length exact for every length (1..8), that changes each direction's cost by
// the same amount, -256 * 840 * (sum of all) + 128^2 * 840 * 64, and only
// differences of costs are used; left out, a cost is at most 840 * 64 * 255^2
// < 2^32.
//
// Line sums are built two at a time: a word whose samples lie on two adjacent
// lines adds to one packed accumulator (at most 8 * 255 per half).  Words that
// start on an even line and on an odd line have accumulators of their own, so
// no word is taken apart; a byte permute lines the two up at the end.
template <int D>
__device__ __forceinline__ uint32_t dir_cost(const uint32_t (&w)[8][4]) {
    static_assert(D >= 0 && D < 8, "direction");
    uint32_t cost = 0;
    auto add = [&](uint32_t sum, int line) {
        if (line >= 0 && line < 15 && dir_weight(D, line)) cost += sum * (sum * (uint32_t)dir_weight(D, line));
    };
    if (dir_word_in_one_line(D)) {
        uint32_t acc[11] = {};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[dir_bin(D, i, 2 * k)] += w[i][k];
#pragma unroll
        for (int l = 0; l < 11; ++l) add((acc[l] * 0x10001u) >> 16, l);  // both halves' sum
        return cost;
    }
    // even[m] holds lines 2m, 2m+1 and odd[m + 1] lines 2m+1, 2m+2, in
    // ascending order of samples for all but direction 4, whose lines descend
    // along a row (the halves then swap roles).
    constexpr bool down = dir_bin(D, 0, 1) < dir_bin(D, 0, 0);
    constexpr int step = dir_row_pair(D) ? 2 : 1;
    uint32_t even[8] = {}, odd[9] = {};
#pragma unroll
    for (int i = 0; i < 8; i += step)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t v = step == 2 ? w[i][k] + w[i + (step - 1)][k] : w[i][k];
            const int low = down ? dir_bin(D, i, 2 * k + 1) : dir_bin(D, i, 2 * k);  // lower line of the two
            if ((low & 1) == 0) even[low >> 1] += v;
            else odd[(low + 1) >> 1] += v;
        }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        // odd[m]: lines 2m-1 and 2m; odd[m + 1]: lines 2m+1 and 2m+2
        const uint32_t x = even[m] + (down ? __byte_perm(odd[m + 1], odd[m], 0x5432)
                                           : __byte_perm(odd[m], odd[m + 1], 0x5432));
        add(down ? x >> 16 : x & 0xFFFFu, 2 * m);
        add(down ? x & 0xFFFFu : x >> 16, 2 * m + 1);
    }
    return cost;
}

// The words of an 8x8 block at `blk` (row pitch in samples, rows 16-byte
// aligned), samples scaled to 8 bits.
__device__ __forceinline__ void dir_load(const uint16_t* blk, int pitch, int shift, uint32_t (&w)[8][4]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint4 row = *reinterpret_cast<const uint4*>(blk + i * pitch);
        w[i][0] = (row.x >> shift) & 0x00FF00FFu;
        w[i][1] = (row.y >> shift) & 0x00FF00FFu;
        w[i][2] = (row.z >> shift) & 0x00FF00FFu;
        w[i][3] = (row.w >> shift) & 0x00FF00FFu;
    }
}

// Costs of directions pair and pair + 4, or of direction d alone.  Fully
// unrolled per direction; the switches are warp-uniform.
template <int P>
__device__ __forceinline__ void dir_costs(const uint16_t* blk, int pitch, int shift, uint32_t& lo, uint32_t& hi) {
    uint32_t w[8][4];
    dir_load(blk, pitch, shift, w);
    lo = dir_cost<P>(w);
    hi = dir_cost<P + 4>(w);
}

__device__ __forceinline__ void dir_costs_pair(int pair, const uint16_t* blk, int pitch, int shift, uint32_t& lo,
                                               uint32_t& hi) {
    switch (pair) {
        case 0: dir_costs<0>(blk, pitch, shift, lo, hi); break;
        case 1: dir_costs<1>(blk, pitch, shift, lo, hi); break;
        case 2: dir_costs<2>(blk, pitch, shift, lo, hi); break;
        default: dir_costs<3>(blk, pitch, shift, lo, hi); break;
    }
}

__device__ __forceinline__ uint32_t dir_cost_of(int d, const uint16_t* blk, int pitch, int shift) {
    uint32_t w[8][4];
    dir_load(blk, pitch, shift, w);
    switch (d) {
        case 0: return dir_cost<0>(w);
        case 1: return dir_cost<1>(w);
        case 2: return dir_cost<2>(w);
        case 3: return dir_cost<3>(w);
        case 4: return dir_cost<4>(w);
        case 5: return dir_cost<5>(w);
        case 6: return dir_cost<6>(w);
        default: return dir_cost<7>(w);
    }
}

// The first direction of the largest cost; cost[d][b] for block b.
__device__ __forceinline__ void best_direction(const uint32_t (*cost)[64], int b, int& best, uint32_t& var) {
    int bd = 0;
    uint32_t top = cost[0][b];
#pragma unroll
    for (int d = 1; d < 8; ++d) {
        const uint32_t c = cost[d][b];
        if (c > top) {
            top = c;
            bd = d;
        }
    }
    best = bd;
    var = (top - cost[(bd + 4) & 7][b]) >> 10;
}

// constrain (src/cdef.rs:126-133); threshold 0 yields 0 for any shift.
__device__ __forceinline__ int constrain(int d, int t, int shift) {
    int a = abs(d);
    int c = min(a, max(0, t - (a >> shift)));
    return d < 0 ? -c : c;
}

__device__ __forceinline__ int ilog2u(unsigned v) { return 31 - __clz(v); }

// adjust_strength (src/cdef.rs:209-220).
__device__ __forceinline__ int adjust_strength(int primary, uint32_t variance) {
    if (variance == 0) return 0;
    uint32_t scaled = variance >> 6;
    uint32_t lg = scaled == 0 ? 0 : min((uint32_t)ilog2u(scaled), 12u);
    return (int)(((uint32_t)primary * (4 + lg) + 8) >> 4);
}

// chroma_direction (src/cdef.rs:224-230).
__device__ __forceinline__ int chroma_direction(int d, int sx, int sy) {
    const uint32_t k10 = 0x66654207u;  // nibbles of [7,0,2,4,5,6,6,6]
    const uint32_t k01 = 0x06432221u;  // nibbles of [1,2,2,2,3,4,6,0]
    if (sx && !sy) return (k10 >> (4 * (d & 7))) & 0xF;
    if (!sx && sy) return (k01 >> (4 * (d & 7))) & 0xF;
    return d & 7;
}

// Per-block filter parameters, offsets in shared-memory samples.
struct BlockFilter {
    int off[6];   // primary d0,d1; secondary (dir+2) d0,d1; secondary (dir+6) d0,d1
    short pri, sec;
    uint8_t pri_shift, sec_shift, pt0, pt1;
};

__device__ __forceinline__ BlockFilter make_filter(int dir, int pri, int sec, int damping, int shift, int pitch) {
    BlockFilter f;
    f.off[0] = dir_offset<0>(dir, pitch);
    f.off[1] = dir_offset<1>(dir, pitch);
    f.off[2] = dir_offset<0>((dir + 2) & 7, pitch);
    f.off[3] = dir_offset<1>((dir + 2) & 7, pitch);
    f.off[4] = dir_offset<0>((dir + 6) & 7, pitch);
    f.off[5] = dir_offset<1>((dir + 6) & 7, pitch);
    f.pri = (short)pri;
    f.sec = (short)sec;
    f.pri_shift = (uint8_t)(pri ? max(0, damping - ilog2u(pri)) : 0);
    f.sec_shift = (uint8_t)(sec ? max(0, damping - ilog2u(sec)) : 0);
    bool odd = ((pri >> shift) & 1) != 0;
    f.pt0 = odd ? 3 : 4;
    f.pt1 = odd ? 3 : 2;
    return f;
}

// One output sample of filter_block (src/cdef.rs:167-202) at smem position s.
__device__ __forceinline__ int filter_px(const uint16_t* s, const BlockFilter& f) {
    const int cur = s[0];
    int mn = cur, mx = cur, sum = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int ptap = k ? f.pt1 : f.pt0;
        const int stap = 2 - k;
        int p0 = s[f.off[k]], p1 = s[-f.off[k]];
        int s0 = s[f.off[2 + k]], s1 = s[-f.off[2 + k]];
        int s2 = s[f.off[4 + k]], s3 = s[-f.off[4 + k]];
        mn = min(mn, min(min(p0, p1), min(min(s0, s1), min(s2, s3))));
        mx = max(mx, max(max(p0 & kMaxMask, p1 & kMaxMask),
                         max(max(s0 & kMaxMask, s1 & kMaxMask), max(s2 & kMaxMask, s3 & kMaxMask))));
        sum += ptap * (constrain(p0 - cur, f.pri, f.pri_shift) + constrain(p1 - cur, f.pri, f.pri_shift));
        sum += stap * (constrain(s0 - cur, f.sec, f.sec_shift) + constrain(s1 - cur, f.sec, f.sec_shift) +
                       constrain(s2 - cur, f.sec, f.sec_shift) + constrain(s3 - cur, f.sec, f.sec_shift));
    }
    int v = cur + ((8 + sum - (sum < 0)) >> 4);
    return min(max(v, mn), mx);
}


}  // namespace cdefk
}  // namespace vaco

namespace vaco {
namespace cdefk {

// ---------------------------------------------------------------- two pixels per register
//
// filter_px() for a horizontal pair of pixels held as two 16-bit lanes of one
// 32-bit word (low lane = left pixel).  Two forms with equal results: one in
// 16-bit integers (any bit depth) and one in half-precision arithmetic that
// is exact for samples of up to 10 bits (see HalfBlock).
__device__ __forceinline__ uint32_t vmin2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t vmax2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t vmins2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("min.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t vmaxs2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// Minimum and maximum over the available taps: the sentinel is the largest
// value to an unsigned minimum and negative to a signed maximum, so neither
// ever picks it (samples are below 2^12).
__device__ __forceinline__ void tap_range(uint32_t v, uint32_t& mn, uint32_t& mx) {
    mn = vmin2(mn, v);
    mx = vmaxs2(mx, v);
}
static_assert(kSent > 0x0FFF && (kSent & 0x8000), "tap_range relies on it");

// Which tap sets a tile's blocks use.  vaco's filter_block clamps the result
// to the min/max of every available tap, but when only one tap set has a
// non-zero strength that clamp never binds: the set's weights sum to 12 <= 16
// and |constrain(d)| <= |d|, so cur + Round(sum/16) stays inside the taps'
// range (for sum > 0: (8 + 12 D) >> 4 <= D for every D >= 0, D = max - cur;
// for sum < 0: (7 - 12 E) >> 4 >= -E, E = cur - min).  A zero strength also
// makes every constrain() of its set 0.  So the taps of a set whose preset
// strength is zero are skipped altogether (pri_on / sec_on, uniform over a
// tile), bit-exactly: the clamp over the remaining set is a no-op.
//
// The taps of filter_pair() are 12 functions of the row's word offset, in the
// order +off[0], -off[0], +off[1], ...: primary d0, d1, then dir+2 d0, d1,
// then dir+6 d0, d1.

// ---- integer form
//
// Every per-lane quantity stays in [0, 65535], so plain 32-bit adds and
// subtracts never carry or borrow across lanes:
//   hi = max(v, cur), |d| = hi - min(v, cur), d+ = hi - cur
//   c  = max(min(|d|, t - (|d| >> s)), 0), c+ = min(c, d+)  (constrain and its
//        positive part; t - x is formed as (t + 1) + ~x, one fused
//        add-min-clamp on signed lanes.  A sentinel's |d| is above 2^15, i.e.
//        negative there, which clamps to the 0 it has to give)
//   acc+ += tap * c+, acc += tap * c        (each <= 24 * 240 = 5760), and
//   at the end acc- = acc - acc+ (the negative parts' sum)
// Output: with pos/neg the non-negative parts of acc+ - acc-,
//   r+ = (pos + 8) >> 4, r- = (neg + 8) >> 4  (vaco's signed rounding)
//   out = min(max(cur + r+, mn + r-) - r-, mx) = clamp(cur + r+ - r-, mn, mx).
struct PairBlock {
    int16_t off[6];       // tap offsets (samples): primary d0,d1; dir+2 d0,d1; dir+6 d0,d1
    uint16_t pri, sec;
    uint8_t pri_shift, sec_shift, pt0, pt1;
};

template <class Block>
__device__ __forceinline__ void set_offsets(Block& f, int dir, int pitch) {
    f.off[0] = (int16_t)dir_offset<0>(dir, pitch);
    f.off[1] = (int16_t)dir_offset<1>(dir, pitch);
    f.off[2] = (int16_t)dir_offset<0>((dir + 2) & 7, pitch);
    f.off[3] = (int16_t)dir_offset<1>((dir + 2) & 7, pitch);
    f.off[4] = (int16_t)dir_offset<0>((dir + 6) & 7, pitch);
    f.off[5] = (int16_t)dir_offset<1>((dir + 6) & 7, pitch);
}

__device__ __forceinline__ void make_block(PairBlock& f, int dir, int pri, int sec, int damping, int shift,
                                           int pitch) {
    set_offsets(f, dir, pitch);
    f.pri = (uint16_t)pri;
    f.sec = (uint16_t)sec;
    f.pri_shift = (uint8_t)(pri ? max(0, damping - ilog2u(pri)) : 0);
    f.sec_shift = (uint8_t)(sec ? max(0, damping - ilog2u(sec)) : 0);
    const bool odd = ((pri >> shift) & 1) != 0;
    f.pt0 = odd ? 3 : 4;
    f.pt1 = odd ? 3 : 2;
}

struct PairSet {  // one tap set's strength and shift
    uint32_t t1, mask;
    int s;
    __device__ __forceinline__ PairSet(uint32_t t, int shift)
        : t1((t + 1) * 0x10001u), mask((0xFFFFu >> shift) * 0x10001u), s(shift) {}
};

__device__ __forceinline__ void tap_step(uint32_t v, uint32_t cur, uint32_t ncur, const PairSet& k, uint32_t w,
                                         uint32_t& accp, uint32_t& acct, uint32_t& mn, uint32_t& mx) {
    const uint32_t hi = vmax2(v, cur);
    const uint32_t ad = hi - vmin2(v, cur);
    const uint32_t c = __viaddmin_s16x2_relu(k.t1, ~((ad >> k.s) & k.mask), ad);
    accp += w * __viaddmin_u16x2(hi, ncur, c);
    acct += w * c;
    tap_range(v, mn, mx);
}

// Filters the pair `cur`; tap(k, row) is the pair at tap k, `row` the word
// offset of the current row from the taps' first row.
template <class Taps>
__device__ __forceinline__ uint32_t filter_pair(uint32_t cur, const Taps& tap, int row, const PairBlock& f,
                                                bool pri_on, bool sec_on) {
    const PairSet kp(f.pri, f.pri_shift), ks(f.sec, f.sec_shift);
    const uint32_t ncur = ~cur + 0x00010001u - (((cur & 0xFFFFu) == 0) ? 0x00010000u : 0u);  // -cur per lane
    uint32_t accp = 0, acct = 0, mn = cur, mx = cur;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t wp = k ? f.pt1 : f.pt0, ws = 2 - k;
        if (pri_on) {
            tap_step(tap(2 * k, row), cur, ncur, kp, wp, accp, acct, mn, mx);
            tap_step(tap(2 * k + 1, row), cur, ncur, kp, wp, accp, acct, mn, mx);
        }
        if (sec_on) {
            tap_step(tap(4 + 2 * k, row), cur, ncur, ks, ws, accp, acct, mn, mx);
            tap_step(tap(4 + 2 * k + 1, row), cur, ncur, ks, ws, accp, acct, mn, mx);
            tap_step(tap(8 + 2 * k, row), cur, ncur, ks, ws, accp, acct, mn, mx);
            tap_step(tap(8 + 2 * k + 1, row), cur, ncur, ks, ws, accp, acct, mn, mx);
        }
    }
    const uint32_t accn = acct - accp;
    const uint32_t both = vmin2(accp, accn);
    const uint32_t rp = ((accp - both + 0x00080008u) >> 4) & 0x0FFF0FFFu;
    const uint32_t rn = ((accn - both + 0x00080008u) >> 4) & 0x0FFF0FFFu;
    return vmin2(vmax2(cur + rp, mn + rn) - rn, mx);
}

// ---- half-precision form, samples of up to 10 bits
//
// The bits of a 16-bit integer n <= 2048 are those of the half-precision
// number n 2^-24: up to 1023 as a subnormal, then as the first normal numbers,
// which have the same spacing.  So a word of two samples is a pair of halves
// as it is, in units of 2^-24, and sums and differences are exact while they
// stay within 2048 units.  Per tap, with s the set's shift and t its strength:
//   d  = v - cur                       exact
//   e  = 2 |d| + (1 - 2^s)             exact (at most 2047)
//   m  = max(t - e / 2^(s+1), 0)       one fused multiply-add, which rounds to
//        whole units: with |d| = q 2^s + r, e / 2^(s+1) = q + (2r + 1 - 2^s) /
//        2^(s+1), whose fraction lies strictly inside (-1/2, 1/2), so m is
//        max(t - (|d| >> s), 0) for every |d|
//   c  = min(|d|, m) with d's sign     constrain(d)
//   acc += tap * c                     exact (at most 12 * 60 + 12 * 16 = 912)
// Four of these run on the FMA pipe and, with the min and max of the taps,
// three on the ALU pipe (the absolute values are operand modifiers), against
// about eleven mostly on the ALU pipe in integers.  A shift of 10 or more
// makes |d| >> s zero for every |d| < 1024, as a shift of 10 does.  The
// sentinel reads as -2.0, far above 2^11 units: m is 0 for every s <= 10.
// The fused kernel took 145 us and 100.7 M warp instructions per 4K 10-bit
// frame with integer taps, 115 us and 78.4 M with these.
struct __align__(16) HalfBlock {
    uint32_t pt, pk1, pk2;  // primary set: t, 1 - 2^s, -2^-(s+1), both lanes
    uint32_t st, sk1, sk2;  // secondary set
    uint32_t w0, w1;        // primary tap weights at distances 1 and 2
    int16_t off[6];
};

__device__ __forceinline__ uint32_t h2(uint32_t bits) { return bits * 0x10001u; }

__device__ __forceinline__ void half_set(int t, int s, uint32_t& ht, uint32_t& k1, uint32_t& k2) {
    s = min(s, 10);
    ht = h2((uint32_t)t);
    k1 = s ? h2(0x8000u | ((1u << s) - 1)) : 0u;   // -(2^s - 1) units
    k2 = h2(0x8000u | (uint32_t)(14 - s) << 10);   // -2^-(s+1): exponent 15 - (s + 1)
}

__device__ __forceinline__ void make_block(HalfBlock& f, int dir, int pri, int sec, int damping, int shift,
                                           int pitch) {
    set_offsets(f, dir, pitch);
    half_set(pri, pri ? max(0, damping - ilog2u(pri)) : 0, f.pt, f.pk1, f.pk2);
    half_set(sec, sec ? max(0, damping - ilog2u(sec)) : 0, f.st, f.sk1, f.sk2);
    const bool odd = ((pri >> shift) & 1) != 0;
    f.w0 = odd ? 0x42004200u : 0x44004400u;  // 3.0 : 4.0
    f.w1 = odd ? 0x42004200u : 0x40004000u;  // 3.0 : 2.0
}

__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hsub2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t hfma2_relu(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.relu.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t habs2(uint32_t a) {
    uint32_t d;
    asm("abs.f16x2 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ uint32_t hmin2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("min.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__device__ __forceinline__ void tap_step_h(uint32_t v, uint32_t cur, uint32_t t, uint32_t k1, uint32_t k2, uint32_t w,
                                           uint32_t& acc, uint32_t& mn, uint32_t& mx) {
    const uint32_t d = hsub2(v, cur);
    const uint32_t e = hfma2(habs2(d), 0x40004000u, k1);
    const uint32_t c = hmin2(habs2(d), hfma2_relu(e, k2, t));
    acc = hfma2(c | (d & 0x80008000u), w, acc);
    tap_range(v, mn, mx);
}

template <class Taps>
__device__ __forceinline__ uint32_t filter_pair(uint32_t cur, const Taps& tap, int row, const HalfBlock& f,
                                                bool pri_on, bool sec_on) {
    uint32_t acc = 0, mn = cur, mx = cur;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t wp = k ? f.w1 : f.w0, ws = k ? 0x3C003C00u : 0x40004000u;  // 1.0 : 2.0
        if (pri_on) {
            tap_step_h(tap(2 * k, row), cur, f.pt, f.pk1, f.pk2, wp, acc, mn, mx);
            tap_step_h(tap(2 * k + 1, row), cur, f.pt, f.pk1, f.pk2, wp, acc, mn, mx);
        }
        if (sec_on) {
            tap_step_h(tap(4 + 2 * k, row), cur, f.st, f.sk1, f.sk2, ws, acc, mn, mx);
            tap_step_h(tap(4 + 2 * k + 1, row), cur, f.st, f.sk1, f.sk2, ws, acc, mn, mx);
            tap_step_h(tap(8 + 2 * k, row), cur, f.st, f.sk1, f.sk2, ws, acc, mn, mx);
            tap_step_h(tap(8 + 2 * k + 1, row), cur, f.st, f.sk1, f.sk2, ws, acc, mn, mx);
        }
    }
    // (8 + sum - (sum < 0)) >> 4 is (|sum| + 8) >> 4 with the sum's sign.  A
    // result below zero is negative as a signed lane too, so the signed max
    // with mn >= 0 clamps it.
    const uint32_t r = (((acc & 0x7FFF7FFFu) + 0x00080008u) >> 4) & 0x07FF07FFu;
    return vmins2(vmaxs2(hadd2(cur, r | (acc & 0x80008000u)), mn), mx);
}

}  // namespace cdefk
}  // namespace vaco
