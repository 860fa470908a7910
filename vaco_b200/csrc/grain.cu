// grain.cu -- AV1 film grain synthesis (spec 7.18.3) on sm_100a.
//
// vaco parses film_grain_params() (crates/codec/vaco-codec-av1/src/
// frame_header.rs:1125-1210) and stops there: grain synthesis is the next
// step after the post-filters.  This file adds it as two kernels.
//
//   grain_template_kernel  one CTA per frame: the per-stripe random block
//       offsets, the three grain templates (82 x 73 luma, up to 82 x 73 per
//       chroma plane) from the caller's Gaussian table, their auto-regressive
//       filtering, and the scaling function of every sample value, written to
//       a small workspace.
//       - The templates' random indices come from the spec's 16-bit LFSR.
//         Each thread takes 32 consecutive samples and starts from the
//         register value 32 c steps in, which it computes from the seed by
//         GF(2) matrix products with M^(32 * 2^b) (M = one LFSR step; the
//         host builds those nine matrices), so the sequence needs no
//         serial walk.
//       - The AR filter is a wavefront over blocks of four columns; see
//         ar_wavefront().
//   grain_apply_kernel  the noise of every output sample straight from the
//       templates in shared memory: the block's offsets pick the template
//       window, the left block's window gives the horizontal overlap and the
//       stripe above the vertical one (the spec's NoiseStripe / NoiseImage
//       values), then the scaling lookup, the chroma merge with the
//       co-located luma and the clip.
//
// Samples above the bit depth would index past the scaling table; they are
// reported (VACO_AV1_MSG_FG_SAMPLE) and the index is clamped.
#include <atomic>
#include <cstring>

#include "common.cuh"
#include "kernels.cuh"

namespace vaco {

namespace {

// A template in shared memory and in the workspace: sample (y, x) at
// [y * kPitch + x + 1].  The shift by one puts the first filtered column
// (x = 3) and every fourth after it on an 8-byte boundary, and the apply
// kernel's luma windows (which start on odd x) on a word boundary.
constexpr int kTW = 82, kTH = 73;  // luma template width / height (chroma uses a corner when subsampled)
constexpr int kPitch = 84;
constexpr int kPlane = 74 * kPitch;  // samples per plane, a multiple of 16 bytes
constexpr int kGrainThreads = 384;   // a run of every plane of a 4:2:0 frame at once
constexpr int kRun = 32;             // template samples a thread draws
constexpr int kApplyThreads = 256;
constexpr int kApplyRows = 2;        // rows of an apply work item

struct GrainLayout {  // workspace offsets in bytes: templates, then scaling entries per plane, then block offsets
    size_t scale, offsets;
};
__host__ __device__ constexpr GrainLayout grain_layout(int np) {
    return GrainLayout{sizeof(int16_t) * kPlane * (size_t)np, sizeof(int16_t) * kPlane * (size_t)np + 8192u * (size_t)np};
}

struct TemplateArgs {
    vaco_av1_film_grain_params p;
    __align__(16) int16_t gauss[2048];
    uint16_t jump[9][16];  // columns of M^(kRun * 2^b)
    int bd, sub_x, sub_y, np;
    int nstripes, nbx;
    unsigned char* workspace;
};

__device__ __forceinline__ int round2(int x, int n) { return n == 0 ? x : (x + (1 << (n - 1))) >> n; }

// One LFSR step of get_random_number (7.18.3.2).
__device__ __forceinline__ unsigned lfsr_step(unsigned r) {
    const unsigned bit = (r ^ (r >> 1) ^ (r >> 3) ^ (r >> 12)) & 1u;
    return (r >> 1) | (bit << 15);
}

__device__ __forceinline__ unsigned gf2_apply(const uint16_t* col, unsigned v) {
    unsigned r = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) r ^= ((v >> i) & 1u) ? col[i] : 0u;
    return r;
}

__device__ __forceinline__ void bar_named(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Packed 16-bit operations with instructions of their own.
__device__ __forceinline__ uint32_t maxs2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t minu2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__device__ __forceinline__ int lo16(uint32_t w) { return (int)(int16_t)(w & 0xFFFFu); }
__device__ __forceinline__ int hi16(uint32_t w) { return (int)w >> 16; }

// The seven taps of the row d above (d = 1..3), columns x-3 .. x+3, as signed
// bytes for dp2a on words of two samples: `even` for a window that starts on
// an even stored column, `odd` for one that starts on an odd one.  Taps past
// the lag are zero.
struct RowTaps {
    uint32_t even[2], odd[2];
};
__device__ __forceinline__ RowTaps row_taps(const uint8_t* coef, int lag, int d) {
    uint32_t c[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int o = k - 4;  // column offset x + o; k = 0 and 8 are padding
        const bool in = d <= lag && o >= -lag && o <= lag;
        c[k] = in ? (uint32_t)(uint8_t)(coef[(lag - d) * (2 * lag + 1) + o + lag] - 128) : 0u;
    }
    RowTaps t;
    t.even[0] = c[1] | c[2] << 8 | c[3] << 16 | c[4] << 24;
    t.even[1] = c[5] | c[6] << 8 | c[7] << 16;
    t.odd[0] = c[1] << 8 | c[2] << 16 | c[3] << 24;
    t.odd[1] = c[4] | c[5] << 8 | c[6] << 16 | c[7] << 24;
    return t;
}

// Dot products of two, three or four words of a window with the first taps of
// it.  For a block's outputs k = 0..3, stored at columns 4b + 4 + k, with w[0..5]
// the row's stored columns 4b .. 4b + 11: w[0..3] with the odd taps, w[1..4]
// with the even ones, w[1..4] with the odd ones, w[2..5] with the even ones.
__device__ __forceinline__ int dot2(uint32_t a, uint32_t b, const uint32_t (&t)[2], int acc) {
    return __dp2a_hi((int)b, (int)t[0], __dp2a_lo((int)a, (int)t[0], acc));
}
__device__ __forceinline__ int dot3(uint32_t a, uint32_t b, uint32_t c, const uint32_t (&t)[2], int acc) {
    return __dp2a_lo((int)c, (int)t[1], dot2(a, b, t, acc));
}
__device__ __forceinline__ int dot4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, const uint32_t (&t)[2], int acc) {
    return __dp2a_hi((int)d, (int)t[1], dot3(a, b, c, t, acc));
}

// Auto-regression (7.18.3.3) of all planes in place in shared memory, as one
// wavefront over blocks of four columns.  An output reads up to three rows
// above, columns x-3 .. x+3, and three samples to its left; row yy filters
// block b at step every * b + row_lag * yy + delay:
//   luma    b + 2 yy: the row above finished block b + 1 one step before;
//   chroma  every = 2 with horizontal subsampling (a block spans two luma
//           blocks), row by row the larger of luma's 2 << sub_y steps and
//           every + 1, behind the luma it reads.
// Only about ten rows of a plane are under way at a time, so a lane takes every
// tenth or so row, and the lanes of all planes fit one warp.  Four warps, one
// per scheduler, each do a part of every block:
//   near  the row above's newest block, the left neighbours, the store: four
//         samples, each of which waits for its left neighbour's clamped value;
//   far   one step ahead: the taps of row y-2, the samples scaled by the
//         filter's shift and the rounding term (0), the taps of row y-3 (1),
//         the taps of row y-1 on the columns it finished two steps before and
//         the co-located luma (2).
// What bounds it is the latency of a step (barrier, load, the chain of four,
// store; 180 ns) times 161 steps of a 4:2:0 frame.  Measured for the whole
// kernel, 4K 4:2:0, lag 3: 45 us; one thread a row, a column a step, chroma
// after luma (526 steps) 171 us; one thread a row and four columns a step,
// every tap by one thread, 62 us; two threads a row 57 us.
struct ArLane {
    const uint8_t* coef = nullptr;  // ar_coeffs_*_plus_128
    int t = 0;                      // the plane's template, an offset into the shared templates
    bool luma = false;              // the plane's filter reads the luma template (at offset 0)
    int rows = 0, cols = 0, sub_x = 0, sub_y = 0;
    int every = 1, start = 0;              // start: step of block 0 of row yy
    int yy = 0, lanes = 1, period = 1;     // the lane's first row, rows to its next one, steps to that
};
struct ArSchedule {
    int every, row_lag, delay, lanes;
    __device__ ArSchedule(bool chroma, int sub_x, int sub_y, int cols) {
        every = chroma ? 1 << sub_x : 1;
        row_lag = chroma ? max(2 << sub_y, every + 1) : 2;
        delay = chroma ? sub_x + 2 * sub_y + 2 : 0;
        lanes = (every * ((cols + 3) / 4 - 1) + row_lag) / row_lag;  // a lane's row ends before its next begins
    }
    __device__ int steps(int rows, int cols) const {
        return row_lag * (rows - 1) + delay + every * ((cols + 3) / 4 - 1) + 1;
    }
};
constexpr int kArWarps = 4;
using ArParts = int4[2][3][32];  // by step parity, far role and lane

// `role` 0: near, 1 .. 3: far 0 .. 2; one warp each.
//
// The near warp's chain works on values biased by -gmin, so the clamp is one
// minimum with a clamp to zero; what the bias adds to the sums is in the
// constants far role 0 starts from.
__device__ __forceinline__ void ar_wavefront(int16_t* S, ArLane L, int role, int lane, int lag, int ar_shift, int gmin,
                                             int range, int steps, ArParts& parts) {
    const unsigned last = (unsigned)(L.every * ((L.cols + 3) / 4 - 1));
    const int odd = L.every - 1;
    int t = -1 - L.start + (role ? 1 : 0);  // steps since block 0 of row yy; far roles are one ahead
    int at = L.t + (3 + L.yy) * kPitch;     // offset of the block's stored columns 4b .. in row yy
    int left = L.cols;                      // columns from the block on
    const int next_row = L.lanes * kPitch;
    auto due = [&]() { return (unsigned)t <= last && (t & odd) == 0; };
    auto done = [&]() { at += 4, left -= 4; };  // a block is
    auto advance = [&]() {
        if (++t == L.period) {
            L.yy += L.lanes;
            t = L.yy < L.rows ? 0 : -(1 << 30);
            at += next_row + left - L.cols;  // blocks done so far: (cols - left) / 4
            left = L.cols;
        }
    };
    if (L.yy >= L.rows) t = -(1 << 30);
    auto words = [&](int d, int k) { return *reinterpret_cast<const uint2*>(S + at - d * kPitch + 4 * k); };
    int c[4];  // left taps at distances 1..3
#pragma unroll
    for (int k = 1; k <= 3; ++k) c[k] = k <= lag ? (int)L.coef[lag * (2 * lag + 1) + lag - k] - 128 : 0;
    if (role == 0) {
        const RowTaps t1 = row_taps(L.coef, lag, 1);
        const uint32_t bias = ((uint32_t)gmin & 0xFFFFu) * 0x10001u;
        int4* q = &parts[1][0][lane];  // step -1
        const int flip = (int)(&parts[1][0][0] - &parts[0][0][0]);
        int dir = -flip;
        for (int step = -1; step < steps; ++step) {
            if (due()) {
                const int4 p0 = q[0], p1 = q[32], p2 = q[64];
                const uint2 n = words(1, 2), l = words(0, 0);
                const int l1 = hi16(l.y), l2 = lo16(l.y), l3 = hi16(l.x);
                // n: columns 4b + 8 .. 4b + 11 of the row above, w[4..5] of dot4()
                const int s0 = p0.x + p1.x + p2.x + c[3] * l3 + c[2] * l2 + c[1] * l1;
                const int s1 = __dp2a_hi((int)n.x, (int)t1.even[1], p0.y + p1.y + p2.y) + c[3] * l2 + c[2] * l1;
                const int s2 = __dp2a_hi((int)n.x, (int)t1.odd[1], p0.z + p1.z + p2.z) + c[3] * l1;
                const int s3 = __dp2a_hi((int)n.y, (int)t1.even[1],
                                         __dp2a_lo((int)n.x, (int)t1.even[1], p0.w + p1.w + p2.w));
                const int v0 = __vimin_s32_relu(s0 >> ar_shift, range);
                const int v1 = __vimin_s32_relu((s1 + c[1] * v0) >> ar_shift, range);
                const int v2 = __vimin_s32_relu((s2 + c[2] * v0 + c[1] * v1) >> ar_shift, range);
                const int v3 = __vimin_s32_relu((s3 + c[3] * v0 + c[2] * v1 + c[1] * v2) >> ar_shift, range);
                const uint2 out = make_uint2(add2((uint32_t)(v0 | v1 << 16), bias),
                                             add2((uint32_t)(v2 | v3 << 16), bias));
                uint32_t* o = reinterpret_cast<uint32_t*>(S + at + 4);
                if (left >= 4) {
                    *reinterpret_cast<uint2*>(o) = out;
                } else {  // two columns are filtered (cols is even), the ones past them keep their values
                    o[0] = out.x;
                }
                done();
            }
            advance();
            q += dir, dir = -dir;
            bar_named(1, 32 * kArWarps);
        }
        return;
    }
    const RowTaps taps = row_taps(L.coef, lag, role == 1 ? 2 : role == 2 ? 3 : 1);
    const int cl = L.luma ? (int)L.coef[2 * lag * (lag + 1)] - 128 : 0;
    // co-located luma: offset of the block's first sample, the second row's
    // distance (subsampled vertically, else none: its part is multiplied by 0),
    // Round2's half and shift
    const bool any_luma = __any_sync(0xFFFFFFFFu, cl != 0);
    int luma_at = (3 + (L.yy << L.sub_y)) * kPitch + 4;
    const int luma_row = (L.lanes << L.sub_y) * kPitch, luma_step = 4 << L.sub_x;
    const int second = L.sub_y ? kPitch / 4 : 0, ones = L.sub_y ? 0x0101 : 0;
    const int shift = L.sub_x + L.sub_y, half = shift ? 1 << (shift - 1) : 0;
    // rounding, the bias of the result, and the biased left neighbours' part
    int base[4];
    base[0] = (1 << (ar_shift - 1)) - (gmin << ar_shift);
    base[1] = base[0] + gmin * c[1], base[2] = base[1] + gmin * c[2], base[3] = base[2] + gmin * c[3];
    for (int step = -1; step < steps; ++step) {
        if (due()) {
            int sum[4] = {0, 0, 0, 0};
            if (role == 3) {
                const uint2 w01 = words(1, 0), w23 = words(1, 1);
                if (any_luma) {  // lanes without one add zero
                    const uint2* q = reinterpret_cast<const uint2*>(S + luma_at);
                    const uint2 q0 = q[0], q1 = L.sub_x ? q[1] : q0;
                    const uint2 r0 = q[second], r1 = q[second + 1];
                    if (L.sub_x) {
                        sum[0] = cl * (__dp2a_lo((int)q0.x, 0x0101, __dp2a_lo((int)r0.x, ones, half)) >> shift);
                        sum[1] = cl * (__dp2a_lo((int)q0.y, 0x0101, __dp2a_lo((int)r0.y, ones, half)) >> shift);
                        sum[2] = cl * (__dp2a_lo((int)q1.x, 0x0101, __dp2a_lo((int)r1.x, ones, half)) >> shift);
                        sum[3] = cl * (__dp2a_lo((int)q1.y, 0x0101, __dp2a_lo((int)r1.y, ones, half)) >> shift);
                    } else {
                        sum[0] = cl * lo16(q0.x), sum[1] = cl * hi16(q0.x);
                        sum[2] = cl * lo16(q0.y), sum[3] = cl * hi16(q0.y);
                    }
                }
                sum[0] = dot4(w01.x, w01.y, w23.x, w23.y, taps.odd, sum[0]);
                sum[1] = dot3(w01.y, w23.x, w23.y, taps.even, sum[1]);
                sum[2] = dot3(w01.y, w23.x, w23.y, taps.odd, sum[2]);
                sum[3] = dot2(w23.x, w23.y, taps.even, sum[3]);
            } else {
                const int d = role + 1;
                const uint2 w01 = words(d, 0), w23 = words(d, 1), w45 = words(d, 2);
                if (role == 1) {
                    const uint2 cur = words(0, 1);
                    sum[0] = (lo16(cur.x) << ar_shift) + base[0], sum[1] = (hi16(cur.x) << ar_shift) + base[1];
                    sum[2] = (lo16(cur.y) << ar_shift) + base[2], sum[3] = (hi16(cur.y) << ar_shift) + base[3];
                }
                sum[0] = dot4(w01.x, w01.y, w23.x, w23.y, taps.odd, sum[0]);
                sum[1] = dot4(w01.y, w23.x, w23.y, w45.x, taps.even, sum[1]);
                sum[2] = dot4(w01.y, w23.x, w23.y, w45.x, taps.odd, sum[2]);
                sum[3] = dot4(w23.x, w23.y, w45.x, w45.y, taps.even, sum[3]);
            }
            parts[(step + 1) & 1][role - 1][lane] = make_int4(sum[0], sum[1], sum[2], sum[3]);
            done();
            luma_at += luma_step;
        }
        const int yy = L.yy;
        advance();
        if (L.yy != yy) luma_at += luma_row - luma_step * ((L.cols + 3) / 4);
        bar_named(1, 32 * kArWarps);
    }
}

// Round2 of the co-located filtered luma of chroma template position (y, x).
__device__ __forceinline__ int luma_term(const int16_t* L, int y, int x, int sub_x, int sub_y) {
    const int ly = ((y - 3) << sub_y) + 3, lx = ((x - 3) << sub_x) + 3;
    int l = 0;
    for (int i = 0; i <= sub_y; ++i)
        for (int j = 0; j <= sub_x; ++j) l += L[(ly + i) * kPitch + lx + j + 1];
    return round2(l, sub_x + sub_y);
}

// ScalingLut entry x of a plane (7.18.3.4) from its points.
__device__ int lut_entry(const uint8_t* v, const uint8_t* sc, int n, int x) {
    if (n == 0) return 0;
    if (x < v[0]) return sc[0];
    if (x >= v[n - 1]) return sc[n - 1];
    int i = 0;
    while (x >= v[i + 1]) ++i;
    const int dy = sc[i + 1] - sc[i], dx = v[i + 1] - v[i];
    const int delta = dy * ((65536 + (dx >> 1)) / dx);
    return sc[i] + (((x - v[i]) * delta + 32768) >> 16);
}

// Random block offsets of every stripe (7.18.3.5): the register is re-seeded
// per stripe and steps once per 32-column block.
__device__ __forceinline__ void block_offsets(const TemplateArgs& a, uint8_t* out, int id, int nthreads) {
    for (int s = id; s < a.nstripes; s += nthreads) {
        unsigned r = a.p.grain_seed;
        r ^= ((unsigned)((s * 37 + 178) & 255)) << 8;
        r ^= (unsigned)((s * 173 + 105) & 255);
        uint8_t* o = out + (long)s * a.nbx;
        for (int bx = 0; bx < a.nbx; ++bx) {
            r = lfsr_step(r);
            o[bx] = (uint8_t)((r >> 8) & 255);
        }
    }
}

// The scaling function scale_lut() of every sample value (at most 255, as the
// points' scalings are bytes), times 2^(16 - scaling shift): the high half of
// an entry's product with a noise sample is then the scaled noise.
// `nthreads` threads, `id` this one's, with named barrier 2.
__device__ __forceinline__ void scaling_entries(const TemplateArgs& a, uint8_t (*lut)[256], uint16_t* out, int id,
                                                int nthreads) {
    const vaco_av1_film_grain_params& p = a.p;
    for (int i = id; i < a.np * 256; i += nthreads) {
        const int plane = i >> 8, x = i & 255;
        int v;
        if (plane == 0 || p.chroma_scaling_from_luma) v = lut_entry(p.point_y_value, p.point_y_scaling, p.num_y_points, x);
        else if (plane == 1) v = lut_entry(p.point_cb_value, p.point_cb_scaling, p.num_cb_points, x);
        else v = lut_entry(p.point_cr_value, p.point_cr_scaling, p.num_cr_points, x);
        lut[plane][x] = (uint8_t)v;
    }
    bar_named(2, nthreads);
    const int lshift = a.bd - 8, n = 1 << a.bd;
    for (int i = id; i < a.np * n; i += nthreads) {
        const int plane = i >> a.bd, index = i & (n - 1), x = index >> lshift, rem = index & ((1 << lshift) - 1);
        int v = lut[plane][x];
        if (lshift && x < 255) v += round2(((int)lut[plane][x + 1] - v) * rem, lshift);
        out[plane * 4096 + index] = (uint16_t)(v << (8 - p.grain_scaling_minus_8));
    }
}

__global__ void __launch_bounds__(kGrainThreads) grain_template_kernel(const __grid_constant__ TemplateArgs a) {
    __shared__ __align__(16) int16_t s_t[3][kPlane];
    __shared__ __align__(16) int16_t s_gauss[2048];
    __shared__ uint8_t s_lut[3][256];
    __shared__ ArParts s_parts;
    // the apply kernel may be scheduled now; it waits for this one to end
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int tid = threadIdx.x;
    const vaco_av1_film_grain_params& p = a.p;
    const GrainLayout layout = grain_layout(a.np);
    const int center = 128 << (a.bd - 8);
    const int gmin = -center, gmax = (256 << (a.bd - 8)) - 1 - center;
    for (int i = tid; i < 256; i += kGrainThreads)
        reinterpret_cast<uint4*>(s_gauss)[i] = reinterpret_cast<const uint4*>(a.gauss)[i];

    __syncthreads();

    // Templates before filtering (7.18.3.3): Round2(Gaussian_Sequence[rand11],
    // shift), kRun samples a thread, all planes at once.
    const int shift = 12 - a.bd + p.grain_scale_shift;
    const int cw = a.sub_x ? 44 : 82, ch = a.sub_y ? 38 : 73;
    const bool cb_on = p.num_cb_points || p.chroma_scaling_from_luma;
    const bool cr_on = p.num_cr_points || p.chroma_scaling_from_luma;
    const int luma_runs = (kTW * kTH + kRun - 1) / kRun, chroma_runs = (cw * ch + kRun - 1) / kRun;
    for (int i = tid; i < luma_runs + (a.np - 1) * chroma_runs; i += kGrainThreads) {
        const int plane = i < luma_runs ? 0 : i < luma_runs + chroma_runs ? 1 : 2;
        const int c = i - (plane == 0 ? 0 : plane == 1 ? luma_runs : luma_runs + chroma_runs);
        const int width = plane ? cw : kTW, n = plane ? cw * ch : kTW * kTH;
        const bool on = plane == 0 ? p.num_y_points > 0 : plane == 1 ? cb_on : cr_on;
        unsigned r = plane == 0 ? p.grain_seed : p.grain_seed ^ (plane == 1 ? 0xb524u : 0x49d8u);
        for (int b = 0; b < 9; ++b)
            if ((c >> b) & 1) r = gf2_apply(a.jump[b], r);
        int y = c * kRun / width, x = c * kRun - y * width;
        for (int k = 0; k < kRun && c * kRun + k < n; ++k) {
            r = lfsr_step(r);
            const int g = on ? s_gauss[(r >> 5) & 2047] : 0;
            s_t[plane][y * kPitch + x + 1] = (int16_t)round2(g, shift);
            if (++x == width) x = 0, ++y;
        }
    }
    __syncthreads();

    // Auto-regression by the first four warps; the others find the block
    // offsets and fill the scaling entries meanwhile.
    const int ar_shift = p.ar_coeff_shift_minus_6 + 6, lag = p.ar_coeff_lag;
    const bool luma_on = p.num_y_points > 0;
    const int rows = ch - 3, cols = cw - 6;
    const int ar_threads = lag == 0 ? 0 : 32 * kArWarps;
    if (tid >= ar_threads) {
        block_offsets(a, a.workspace + layout.offsets, tid - ar_threads, kGrainThreads - ar_threads);
        scaling_entries(a, s_lut, reinterpret_cast<uint16_t*>(a.workspace + layout.scale), tid - ar_threads,
                        kGrainThreads - ar_threads);
    } else {
        const ArSchedule luma(false, 0, 0, 76), chroma(true, a.sub_x, a.sub_y, cols);  // 10 lanes, 5 to 10 a plane
        const int lane = tid & 31;
        const int plane = lane < luma.lanes ? 0 : lane < luma.lanes + chroma.lanes ? 1 : 2;
        const ArSchedule& when = plane ? chroma : luma;
        ArLane L;
        L.t = plane * kPlane;
        L.coef = plane == 0 ? p.ar_coeffs_y_plus_128 : plane == 1 ? p.ar_coeffs_cb_plus_128 : p.ar_coeffs_cr_plus_128;
        L.luma = plane && luma_on;
        L.rows = plane ? rows : 70, L.cols = plane ? cols : 76, L.sub_x = a.sub_x, L.sub_y = a.sub_y;
        L.every = when.every, L.lanes = when.lanes, L.period = when.lanes * when.row_lag;
        L.yy = lane - (plane == 0 ? 0 : plane == 1 ? luma.lanes : luma.lanes + chroma.lanes);
        L.start = when.row_lag * L.yy + when.delay;
        if (L.yy >= when.lanes || plane >= a.np || (plane == 1 && !cb_on) || (plane == 2 && !cr_on)) L.rows = 0;
        int steps = luma.steps(70, 76);
        if (a.np > 1) steps = max(steps, chroma.steps(rows, cols));
        ar_wavefront(s_t[0], L, tid >> 5, lane, lag, ar_shift, gmin, gmax - gmin, steps, s_parts);
    }
    __syncthreads();
    if (lag == 0) {  // no taps but the chroma planes' co-located luma
        for (int i = tid; i < 70 * 76; i += kGrainThreads) {
            int16_t& v = s_t[0][(3 + i / 76) * kPitch + 4 + i % 76];
            v = (int16_t)clampi(v, gmin, gmax);  // Round2(0) added
        }
        __syncthreads();
        for (int i = tid; i < (a.np > 1 ? 2 * rows * cols : 0); i += kGrainThreads) {
            const int pl = 1 + i / (rows * cols), j = i % (rows * cols);
            const int y = 3 + j / cols, x = 3 + j % cols;
            if (!(pl == 1 ? cb_on : cr_on)) continue;
            const int cl = (pl == 1 ? p.ar_coeffs_cb_plus_128[0] : p.ar_coeffs_cr_plus_128[0]) - 128;
            const int sum = luma_on ? cl * luma_term(s_t[0], y, x, a.sub_x, a.sub_y) : 0;
            int16_t& v = s_t[pl][y * kPitch + x + 1];
            v = (int16_t)clampi(v + round2(sum, ar_shift), gmin, gmax);
        }
        __syncthreads();
    }

    for (int i = tid; i < a.np * kPlane / 8; i += kGrainThreads)
        reinterpret_cast<uint4*>(a.workspace)[i] = reinterpret_cast<const uint4*>(s_t[0])[i];
}

struct ApplyArgs {
    vaco_av1_film_grain_params p;
    DevPlaneC in[3];
    DevPlane out[3];
    int bd, sub_x, sub_y, np, w, h, nbx;
    int pw[3], ph[3];
    // work items: kApplyRows rows of an 8-sample chunk, of luma (0) or of both
    // chroma planes (1)
    int chunks_per_row[2];
    unsigned cpr_recip[2];  // fast_div_recip(chunks_per_row)
    int luma_items, items;
    int on[3];              // the plane gets grain
    int chroma_rows;        // template rows a chroma window can reach
    const unsigned char* workspace;
    DeviceStatus* status;
    int vec;  // every plane's rows start 16-byte aligned: 8-sample runs load and store as one vector
};

// Eight samples of a template from stored index i, two a word.
__device__ __forceinline__ void run8(const int16_t* T, int i, uint32_t (&w)[4]) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(T) + (i >> 1);
    if (i & 1) {
        uint32_t a = q[0];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t b = q[k + 1];
            w[k] = __byte_perm(a, b, 0x5432);
            a = b;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = q[k];
    }
}

__device__ __forceinline__ uint32_t pack16(int lo, int hi) { return ((uint32_t)lo & 0xFFFFu) | (uint32_t)hi << 16; }

// Round2(a * wa + b * wb, 5) clamped (7.18.3.5).
__device__ __forceinline__ int overlap(int a, int wa, int b, int wb, int gmin, int gmax) {
    return clampi((a * wa + b * wb + 16) >> 5, gmin, gmax);
}

// Template index of block offset byte `off`'s window.
__device__ __forceinline__ int window_at(int off, int psx, int psy) {
    const int ox = psx ? 6 + (off >> 4) : 9 + 2 * (off >> 4), oy = psy ? 6 + (off & 15) : 9 + 2 * (off & 15);
    return oy * kPitch + ox + 1;
}

// Windows of one stripe at an 8-sample chunk: the block's, and for a block's
// first chunk the window of the block to its left (-1: no overlap).
struct StripeAt {
    int at, left;
    __device__ __forceinline__ explicit StripeAt(const void*) : at(0), left(-1) {}  // a plane without grain
    __device__ __forceinline__ StripeAt(const uint8_t* offsets, int nbx, int s, int x0, int psx, int psy,
                                        bool overlap) {
        const int bx = x0 >> (5 - psx), j0 = x0 - (bx << (5 - psx));
        const uint8_t* o = offsets + (long)s * nbx + bx;
        at = window_at(__ldg(o), psx, psy) + j0;
        left = overlap && bx > 0 && j0 == 0 ? window_at(__ldg(o - 1), psx, psy) + (32 >> psx) : -1;
    }
    // NoiseStripe[s][plane][i][x0 .. x0+7] of 7.18.3.5
    __device__ __forceinline__ void run(const int16_t* T, int i, int psx, int gmin, int gmax, uint32_t (&g)[4]) const {
        run8(T, at + i * kPitch, g);
        if (left >= 0) {
            const int16_t* r = T + left + i * kPitch;
            if (psx)
                g[0] = pack16(overlap(r[0], 23, lo16(g[0]), 22, gmin, gmax), hi16(g[0]));
            else
                g[0] = pack16(overlap(r[0], 27, lo16(g[0]), 17, gmin, gmax),
                              overlap(r[1], 17, hi16(g[0]), 27, gmin, gmax));
        }
    }
};

// Eight samples as four words; past n they read as zero.
struct Run8 {
    uint32_t w[4];
    __device__ __forceinline__ Run8(const uint16_t* src, int n, bool full) {
        if (full) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(src));
            w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                w[k] = (2 * k < n ? (uint32_t)src[2 * k] : 0u) | (2 * k + 1 < n ? (uint32_t)src[2 * k + 1] << 16 : 0u);
        }
    }
    __device__ __forceinline__ uint32_t any() const { return w[0] | w[1] | w[2] | w[3]; }
};

__device__ __forceinline__ void store8(uint16_t* dst, int n, bool full, const uint32_t (&v)[4]) {
    if (full) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k < n) dst[k] = (uint16_t)((k & 1) ? v[k >> 1] >> 16 : v[k >> 1]);
    }
}

// Every plane read once and written once, 49.8 MB for a 4K 10-bit frame.  The
// templates and the scaling entries sit in shared memory (31 KB for 4:2:0 at
// 10 bits), so a CTA walks its share of the frame.  A thread's item is two rows
// of an 8-sample chunk: its windows' positions serve both, neighbouring lanes
// take neighbouring chunks, and U and V share the co-located luma.  Samples
// stay two to a word but for the lookup and the product, whose high half is
// the scaled noise; adding and clamping are one packed add-min and one packed
// max.  A 4K 10-bit frame takes 25 us (43.5 us with the templates read sample by
// sample from L1 and the scaling interpolated per sample), bound by latency and
// issue; four rows an item, or 3, 5 or 6 CTAs per SM, change nothing.
__global__ void __launch_bounds__(kApplyThreads, 4) grain_apply_kernel(const __grid_constant__ ApplyArgs a) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    overlap_prologue();
    const vaco_av1_film_grain_params& p = a.p;
    const int bd = a.bd, maxv = (1 << bd) - 1, lshift = bd - 8;
    // luma template, chroma templates, scaling entries
    const int chroma_plane = a.chroma_rows * kPitch;
    int16_t* const s_t = reinterpret_cast<int16_t*>(s_dyn);
    uint16_t* const s_scale =
        reinterpret_cast<uint16_t*>(s_dyn + sizeof(int16_t) * (kPlane + (a.np > 1 ? 2 * chroma_plane : 0)));
    const GrainLayout layout = grain_layout(a.np);
    if (p.apply_grain) {
        const uint4* src = reinterpret_cast<const uint4*>(a.workspace);
        uint4* dst = reinterpret_cast<uint4*>(s_dyn);
        const int nl = kPlane / 8, nc = chroma_plane / 8, ns = 1 << (bd - 3);
        for (int i = threadIdx.x; i < nl; i += kApplyThreads) dst[i] = __ldg(src + i);
        for (int k = 1; k < a.np; ++k)
            for (int i = threadIdx.x; i < nc; i += kApplyThreads) dst[nl + (k - 1) * nc + i] = __ldg(src + k * nl + i);
        for (int k = 0; k < a.np; ++k)
            for (int i = threadIdx.x; i < ns; i += kApplyThreads)
                reinterpret_cast<uint4*>(s_scale)[k * ns + i] =
                    __ldg(reinterpret_cast<const uint4*>(a.workspace + layout.scale + k * 8192) + i);
    }
    __syncthreads();
    const uint8_t* const offsets = a.workspace + layout.offsets;
    const int center = 128 << lshift, gmin = -center, gmax = (256 << lshift) - 1 - center;
    int min_v = 0, max_luma = (256 << lshift) - 1, max_chroma = max_luma;
    if (p.clip_to_restricted_range) {
        min_v = 16 << lshift;
        max_luma = 235 << lshift;
        max_chroma = p.mc_identity ? max_luma : 240 << lshift;
    }
    const uint32_t lo2 = pack16(min_v, min_v), max2 = pack16(maxv, maxv);
    // Two samples of a word plus their scaled noise; the entries e0, e1 are
    // those of the samples' scaling indices.  (Round2 by the scaling shift of
    // entry * g is (entry << (16 - shift)) * g + 2^15, high half.)
    auto grained = [&](uint32_t orig, int e0, int e1, uint32_t g, uint32_t hi2) {
        const uint32_t n0 = (uint32_t)(e0 * lo16(g) + 0x8000), n1 = (uint32_t)(e1 * hi16(g) + 0x8000);
        return maxs2(__viaddmin_s16x2(orig, __byte_perm(n0, n1, 0x7632), hi2), lo2);
    };
    // NoiseImage[plane][y][x0 .. x0+7]: the stripe's run with the vertical
    // overlap against the stripe above on the stripe's first rows.
    auto noise = [&](const int16_t* T, const StripeAt& here, int psx, int psy, int s, int i, int x0,
                     uint32_t (&g)[4]) {
        here.run(T, i, psx, gmin, gmax, g);
        if (p.overlap_flag && s > 0 && (psy ? i == 0 : i < 2)) {
            uint32_t gp[4];
            const StripeAt above(offsets, a.nbx, s - 1, x0, psx, psy, true);
            above.run(T, i + (32 >> psy), psx, gmin, gmax, gp);
            const int wo = psy ? 23 : i == 0 ? 27 : 17, wn = psy ? 22 : i == 0 ? 17 : 27;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                g[k] = pack16(overlap(lo16(gp[k]), wo, lo16(g[k]), wn, gmin, gmax),
                              overlap(hi16(gp[k]), wo, hi16(g[k]), wn, gmin, gmax));
        }
    };
    const uint32_t above_depth = ~max2;
    auto check = [&](const Run8& v, int plane, int y, int x0) {
        if (v.any() & above_depth)
            report_error(a.status, STAGE_GRAIN, ((unsigned long long)plane << 44) | ((unsigned long long)y << 20) | x0,
                         VACO_AV1_MSG_FG_SAMPLE);
    };
    const uint32_t hi_luma = pack16(max_luma, max_luma), hi_chroma = pack16(max_chroma, max_chroma);
    for (int item = blockIdx.x * kApplyThreads + threadIdx.x; item < a.items; item += gridDim.x * kApplyThreads) {
        const bool chroma = item >= a.luma_items;
        const int j = chroma ? item - a.luma_items : item;
        const int cpr = a.chunks_per_row[chroma];
        const int rp = (int)fast_div(j, cpr, a.cpr_recip[chroma]), x0 = (j - rp * cpr) * 8, y0 = rp * kApplyRows;
        if (!chroma) {
            const int n = min(8, a.pw[0] - x0);
            const bool full = n == 8 && a.vec, grain = p.apply_grain && a.on[0];
            const int s = y0 >> 5;
            const uint16_t* src = a.in[0].data + (long)y0 * a.in[0].stride + x0;
            // both rows' loads before the first is used
            const bool two = y0 + 1 < a.ph[0];
            const Run8 row0(src, n, full), row1(two ? src + a.in[0].stride : src, n, full);
            const StripeAt here = grain ? StripeAt(offsets, a.nbx, s, x0, 0, 0, p.overlap_flag) : StripeAt(s_dyn);
            auto one = [&](const Run8& orig, int y) {
                check(orig, 0, y, x0);
                uint32_t v[4] = {orig.w[0], orig.w[1], orig.w[2], orig.w[3]};
                if (grain) {
                    uint32_t g[4];
                    noise(s_t, here, 0, 0, s, y - (s << 5), x0, g);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        // only a sample above the bit depth, which is reported, is cut
                        const uint32_t i = minu2(v[k], max2);
                        v[k] = grained(v[k], s_scale[i & 0xFFFFu], s_scale[i >> 16], g[k], hi_luma);
                    }
                }
                store8(a.out[0].data + (long)y * a.out[0].stride + x0, n, full, v);
            };
            one(row0, y0);
            if (two) one(row1, y0 + 1);
            continue;
        }
        const int n = min(8, a.pw[1] - x0);
        const bool full = n == 8 && a.vec, grain = p.apply_grain && (a.on[1] || a.on[2]);
        const int s = y0 >> (5 - a.sub_y);
        const StripeAt here = grain ? StripeAt(offsets, a.nbx, s, x0, a.sub_x, a.sub_y, p.overlap_flag)
                                    : StripeAt(s_dyn);
#pragma unroll 1
        for (int y = y0; y < min(y0 + kApplyRows, a.ph[1]); ++y) {
            const Run8 orig_u(a.in[1].data + (long)y * a.in[1].stride + x0, n, full);
            const Run8 orig_v(a.in[2].data + (long)y * a.in[2].stride + x0, n, full);
            uint32_t avg[4] = {};  // co-located luma, two a word
            if (grain) {
                const uint16_t* lrow = a.in[0].data + (long)(y << a.sub_y) * a.in[0].stride;
                if (!a.sub_x) {
                    const Run8 l(lrow + x0, n, full);
#pragma unroll
                    for (int k = 0; k < 4; ++k) avg[k] = l.w[k];
                } else if (full && 2 * x0 + 16 <= a.w) {
                    const Run8 l0(lrow + 2 * x0, 8, true), l1(lrow + 2 * x0 + 8, 8, true);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t w0 = k < 2 ? l0.w[2 * k] : l1.w[2 * k - 4];
                        const uint32_t w1 = k < 2 ? l0.w[2 * k + 1] : l1.w[2 * k - 3];
                        // (first + second + 1) >> 1 of both pairs
                        avg[k] = ((__byte_perm(w0, w1, 0x5410) + __byte_perm(w0, w1, 0x7632) + 0x00010001u) >> 1) &
                                 0x7FFF7FFFu;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int lx = min((x0 + k) << 1, a.w - 1), lnx = min(lx + 1, a.w - 1);
                        avg[k >> 1] |= (uint32_t)((__ldg(lrow + lx) + __ldg(lrow + lnx) + 1) >> 1) << (16 * (k & 1));
                    }
                }
            }
            auto one = [&](const Run8& orig, int plane, int mult, int lmult, int offset) {
                check(orig, plane, y, x0);
                uint32_t v[4] = {orig.w[0], orig.w[1], orig.w[2], orig.w[3]};
                if (grain && a.on[plane]) {
                    uint32_t g[4];
                    noise(s_t + kPlane + (plane - 1) * chroma_plane, here, a.sub_x, a.sub_y, s,
                          y - (s << (5 - a.sub_y)), x0, g);
                    const uint16_t* sc = s_scale + (plane << bd);
                    // ((luma * lmult + sample * mult) >> 6) + offset, or the luma alone
                    const int lm = p.chroma_scaling_from_luma ? 64 : lmult - 128;
                    const int cm = p.chroma_scaling_from_luma ? 0 : mult - 128;
                    const int off = p.chroma_scaling_from_luma ? 0 : (offset - 256) << (lshift + 6);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int i0 = ((int)(avg[k] & 0xFFFFu) * lm + (int)(v[k] & 0xFFFFu) * cm + off) >> 6;
                        const int i1 = ((int)(avg[k] >> 16) * lm + (int)(v[k] >> 16) * cm + off) >> 6;
                        v[k] = grained(v[k], sc[__vimin_s32_relu(i0, maxv)], sc[__vimin_s32_relu(i1, maxv)], g[k],
                                       hi_chroma);
                    }
                }
                store8(a.out[plane].data + (long)y * a.out[plane].stride + x0, n, full, v);
            };
            one(orig_u, 1, p.cb_mult, p.cb_luma_mult, p.cb_offset);
            one(orig_v, 2, p.cr_mult, p.cr_luma_mult, p.cr_offset);
        }
    }
}

// Columns of M^(kRun * 2^b), M = one LFSR step, for b = 0..8.
void build_jump(uint16_t (&jump)[9][16]) {
    auto step = [](unsigned r) {
        const unsigned bit = (r ^ (r >> 1) ^ (r >> 3) ^ (r >> 12)) & 1u;
        return (r >> 1) | (bit << 15);
    };
    auto apply = [](const uint16_t* col, unsigned v) {
        unsigned r = 0;
        for (int i = 0; i < 16; ++i)
            if ((v >> i) & 1u) r ^= col[i];
        return r;
    };
    for (int i = 0; i < 16; ++i) {
        unsigned r = 1u << i;
        for (int k = 0; k < kRun; ++k) r = step(r);
        jump[0][i] = (uint16_t)r;
    }
    for (int b = 1; b < 9; ++b)
        for (int i = 0; i < 16; ++i) jump[b][i] = (uint16_t)apply(jump[b - 1], apply(jump[b - 1], 1u << i));
}

}  // namespace

size_t film_grain_workspace_bytes(int np, int w, int h) {
    const size_t nstripes = (size_t)(((h + 1) / 2 + 15) / 16), nbx = (size_t)(((w + 1) / 2 + 15) / 16);
    return grain_layout(np).offsets + nstripes * nbx;
}

cudaError_t launch_grain_template(const vaco_av1_film_grain_params& p, const int16_t* gauss, int np, int bd,
                                  int sub_x, int sub_y, int w, int h, void* workspace, cudaStream_t stream) {
    static thread_local TemplateArgs t;  // 4.6 KB, off the stack; the launch copies it
    t.p = p;
    memcpy(t.gauss, gauss, sizeof t.gauss);
    build_jump(t.jump);
    t.bd = bd, t.sub_x = sub_x, t.sub_y = sub_y, t.np = np;
    t.nstripes = ((h + 1) / 2 + 15) / 16, t.nbx = ((w + 1) / 2 + 15) / 16;
    t.workspace = static_cast<unsigned char*>(workspace);
    return launch_overlapped(grain_template_kernel, dim3(1), dim3(kGrainThreads), 0, stream, t);
}

cudaError_t launch_grain_apply(const vaco_av1_film_grain_params& p, const DevPlaneC* in, const DevPlane* out,
                               int np, int bd, int sub_x, int sub_y, int w, int h, const void* workspace,
                               DeviceStatus* status, int sm_count, cudaStream_t stream) {
    ApplyArgs a;
    memset(&a, 0, sizeof a);
    a.p = p;
    a.bd = bd, a.sub_x = sub_x, a.sub_y = sub_y, a.np = np, a.w = w, a.h = h, a.nbx = ((w + 1) / 2 + 15) / 16;
    a.workspace = static_cast<const unsigned char*>(workspace);
    a.status = status;
    a.on[0] = p.num_y_points > 0;
    a.on[1] = p.num_cb_points > 0 || p.chroma_scaling_from_luma;
    a.on[2] = p.num_cr_points > 0 || p.chroma_scaling_from_luma;
    a.chroma_rows = sub_y ? 38 : 74;
    long long items = 0;
    a.vec = 1;
    for (int k = 0; k < np; ++k) {
        a.in[k] = in[k];
        a.out[k] = out[k];
        a.pw[k] = k ? (w + sub_x) >> sub_x : w;
        a.ph[k] = k ? (h + sub_y) >> sub_y : h;
        a.vec = a.vec && (reinterpret_cast<uintptr_t>(in[k].data) | reinterpret_cast<uintptr_t>(out[k].data)) % 16 == 0 &&
                in[k].stride % 8 == 0 && out[k].stride % 8 == 0;
        if (k > 1) continue;
        a.chunks_per_row[k] = (a.pw[k] + 7) / 8;
        a.cpr_recip[k] = fast_div_recip((unsigned)a.chunks_per_row[k]);
        items += (long long)a.chunks_per_row[k] * ((a.ph[k] + kApplyRows - 1) / kApplyRows);
        if (k == 0) a.luma_items = (int)items;
    }
    // both counts fit an int: at most 65536 x 65536 samples of 16 an item, and
    // the loop's last step past the end adds a grid
    if (items >= (1LL << 30)) return cudaErrorInvalidValue;
    a.items = (int)items;
    if (items == 0) return cudaSuccess;
    const size_t smem = sizeof(int16_t) * (kPlane + (np > 1 ? 2 * a.chroma_rows * kPitch : 0)) + ((size_t)np << (bd + 1));
    // 4:2:2 and 4:4:4 at 12 bits need more than the default limit, up to 62 KB
    static std::atomic<unsigned long long> devices{0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !(devices.load(std::memory_order_acquire) & (1ull << dev))) {
        const cudaError_t e =
            cudaFuncSetAttribute(grain_apply_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
        if (e != cudaSuccess) return e;
        if (dev < 64) devices.fetch_or(1ull << dev, std::memory_order_release);
    }
    constexpr int per_sm = 4;
    const long long want = (items + kApplyThreads - 1) / kApplyThreads;
    const int grid = (int)(want < (long long)sm_count * per_sm ? want : (long long)sm_count * per_sm);
    return launch_overlapped(grain_apply_kernel, dim3(grid), dim3(kApplyThreads), smem, stream, a);
}

}  // namespace vaco
