// dbcdef.cu -- deblocking (AV1 7.14) fused with CDEF (vaco src/decode.rs:739-862)
// in one pass over each 64x64 filter block.
//
// Why fused: the chain needs the deblocked picture only (a) as CDEF's input
// and (b) as restoration's pre-CDEF source, which restoration reads at just
// four rows around every stripe boundary (src/restoration.rs:233-244).  One
// CTA therefore stages its tile with a 16-sample halo, runs both deblocking
// passes in shared memory (all vertical edges of the staged region, then the
// horizontal edges that reach the CDEF window), writes the stripe-boundary
// rows to a compact buffer, and filters CDEF straight from the deblocked tile.
// The deblocked picture never round-trips through HBM.
//
// Halo arithmetic (plane units, tile [x0, x0+tw) x [y0, y0+th)):
//   CDEF reads the deblocked window [x0-2, x0+tw+2) x [y0-2, y0+th+2).
//   An edge of filter size n sits on a multiple of n (7.14.2: it is a
//   transform edge of the block on its q side), and it modifies n/2 samples
//   on either side at most (14-tap: 6, 8-tap: 3, 6-tap: 2, 4-tap: 2).  The
//   edges that reach the window are therefore exactly the 4-aligned ones in
//   [y0, y0+th] (horizontal) and [x0, x0+tw] (vertical); the edge at y0-4,
//   say, is a size-4 edge and stops at y0-3.
//   Those horizontal edges read rows [E-7, E+6] (luma, 14-tap only where E is
//   a multiple of 16) or [E-3, E+2] (chroma, at most 6 taps): rows
//   [y0-7, y0+th+7) for luma and [y0-3, y0+th+3) for chroma, which is where
//   the vertical pass must run.  Vertical edges read columns [X-7, X+6].
// The staged region is [x0-8, x0+tw+8) x [y0-8, y0+th+8).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "cdef_core.cuh"
#include "common.cuh"
#include "deblock_core.cuh"
#include "kernels.cuh"

namespace vaco {

namespace {

using namespace cdefk;
using namespace dbk;

constexpr int kHalo = 8;
// Edge segments (one edge x one 4-sample cell) per pass and plane are at most
// (th/4+4) x (tw/4+1) = 340.  Size-class lists: 0 = size 4 (any plane, up to
// 3 x 340), 1 = chroma size 8 (2 x 340), 2 = luma size 8, 3 = luma size 16.
__constant__ int c_list_off[4] = {0, 1020, 1700, 2040};
constexpr int kListTotal = 2380;
// Rows of the luma CDEF window (th + 4) kept as odd-aligned pairs, and the
// words of luma's and both 4:2:0 chroma planes' (see shift_copy()).
constexpr int kShiftRows = 64 + 4;
constexpr int kShiftWords = kShiftRows * (64 + 2 * kHalo) / 2 + 2 * (32 + 2 * kHalo) * (32 + 2 * kHalo) / 2;

// Side-information window of a tile: cells [mi_r0 - kWinTop, +kWinRows) x
// [mi_c0 - kWinLeft, +kWinCols) of the luma maps, and the same shape around
// the tile's own cell origin in the chroma transform map.  Relative to the
// tile, the two passes read transform sizes at cell rows [-2, 17] and
// columns [-1, 16] (previous cells included), and subsampled chroma reads
// levels at luma cells up to row and column 17.
constexpr int kWinTop = 3, kWinLeft = 2, kWinRows = 22, kWinCols = 20, kWinCells = kWinRows * kWinCols;
struct SideWindow {
    uint8_t tx[2][kWinCells];  // luma, chroma transform sizes: log2 width | log2 height << 4
    uint32_t lvl[kWinCells];   // loop-filter levels (Yv, Yh, U, V) when a level map is given
};
__device__ __forceinline__ uint8_t tx_logs(int t) { return (uint8_t)(tx_w_log2(t) | tx_h_log2(t) << 4); }

// n / d for the tile loops' small quotients (segments per edge row 9, 10,
// 17, 18; 16-byte vectors per staged row 6, 10; sentinel window widths 36,
// 68) as one multiply and shift: with m = ceil(2^20 / d), (n m) >> 20 is
// n / d for 0 <= n < 2^20 / d, which every loop here stays under (n is at
// most 80 x 10, 20 x 18 or 68 x 68).  m is computed once per loop.
__device__ __forceinline__ unsigned small_div_magic(int d) { return ((1u << 20) + (unsigned)d - 1) / (unsigned)d; }
__device__ __forceinline__ int small_div(int n, unsigned m) { return (int)(((unsigned)n * m) >> 20); }

struct PlaneGeom {
    int tw, th;        // tile extent in this plane
    int pitch, rows;   // staged region
    int sx, sy;
};

__device__ __forceinline__ PlaneGeom plane_geom(int p, int ssx, int ssy) {
    PlaneGeom g;
    g.sx = p ? ssx : 0;
    g.sy = p ? ssy : 0;
    g.tw = 64 >> g.sx;
    g.th = 64 >> g.sy;
    g.pitch = g.tw + 2 * kHalo;
    g.rows = g.th + 2 * kHalo;
    return g;
}

struct DbCdefArgs {
    DevPlaneC src[3];
    DevPlane dst[3];            // CDEF output planes
    DevPlane pre_rows[3];       // stripe-boundary rows of the deblocked picture (may be null)
    int num_planes, ssx, ssy, bit_depth, shift;
    int mi_rows, mi_cols, coded_width, coded_height;
    // deblocking
    const uint8_t* tx_luma;
    const uint8_t* tx_chroma;
    const uint8_t* lvl_map;
    uint8_t levels[4];
    int sharpness;
    int deblock_on;
    // CDEF
    int cdef_on;
    const uint8_t* skip;
    const int32_t* cdef_idx;
    int cdef_stride, cdef_count;
    int damping;
    uint8_t y_pri[8], y_sec[8], uv_pri[8], uv_sec[8];
    DeviceStatus* status;
    int vec_ok;
    int dst_vec;                // the CDEF planes' rows start 16-byte aligned
    int staged_vectors;         // 16-byte vectors of all staged planes together
    DirectPlane direct[3];      // final output written here too (see DirectPlane)
    size_t plane_off[3];        // shared-memory offset (samples) of each staged plane
    int tile_row0;              // first row of tiles of a per-frame launch
};

// The taps of one lane as words of the staged plane: a pair that starts on an
// even sample is one aligned word of the plane, one that starts on an odd
// sample one word of a copy shifted by one sample.
struct WordTaps {
    const uint32_t* w[12];
    __device__ __forceinline__ uint32_t operator()(int k, int row) const { return w[k][row]; }
};
// The same without a shifted copy: two aligned words and a byte permute.
struct PairTaps {
    const uint32_t* w[12];  // aligned word holding sample i & ~1
    uint32_t sel[12];       // 0x3210 (i even) or 0x5432 (i odd)
    __device__ __forceinline__ uint32_t operator()(int k, int row) const {
        return __byte_perm(w[k][row], w[k][row + 1], sel[k]);
    }
};

// CDEF output of block row br of planes p0 .. p0 + NPL - 1 (both chroma planes
// share their blocks' parameters) from the staged (deblocked) samples `t` of
// plane p0; the next plane's are `plane_words` words on.  One warp; lane l
// owns pixel pairs at tile column 2*(l % ppr), rows l / ppr + RPI*j.  PITCH is
// the staged pitch, BH the block height.
// pri_on / sec_on: the tile preset's primary / secondary strength is
// non-zero; with neither, every sample stays as it is.
// SHIFT: the pairs that start on odd samples are at s1, rows from row kHalo-2
// on the staged pitch, planes at the same distance.
// PARTS warps share the block row, by plane first, then by rows; `part` is
// this warp's share.
template <int PITCH, int BH, int RPI, int NPL, int PARTS, bool SHIFT, bool DIRECT, class Block>
__device__ __forceinline__ void filter_block_row(const DbCdefArgs& a, int p0, const uint16_t* t, const uint32_t* s1,
                                                 int plane_words, int px0, int py0, const uint8_t* active,
                                                 const Block* blocks, bool pri_on, bool sec_on, int br, int part,
                                                 int lane, int sx) {
    constexpr int ppr = 32 / RPI;          // pairs per row: the tile is 2 ppr samples wide
    constexpr bool by_plane = PARTS >= NPL;
    constexpr int row_parts = by_plane ? PARTS / NPL : 1, steps = BH / RPI / row_parts;
    static_assert(steps >= 1, "every warp has a row");
    const int pl0 = by_plane ? part % NPL : 0, pl1 = by_plane ? pl0 + 1 : NPL;
    const int j0 = by_plane ? part / NPL * steps : 0;
    const int x = 2 * (lane % ppr), lr = lane / ppr;
    const int r0 = br * BH;
    const int gx = px0 + x;
    const int width = a.dst[p0].width, height = a.dst[p0].height;
    if (py0 + r0 >= height) return;
    const bool col_in = gx < width;
    const int rows_here = min(BH, height - (py0 + r0));
    const int b = br * 8 + (x >> (3 - sx));
    const int base_i = (kHalo + r0 + lr) * PITCH + kHalo + x;  // left sample, first row of this lane
    const uint32_t* t32 = reinterpret_cast<const uint32_t*>(t);
    const uint32_t* cw = t32 + (base_i >> 1);
    // Runs out(word offset, value) over the lane's rows of every plane.
    auto rows = [&](auto&& value) {
#pragma unroll 1  // smaller code: the fused kernel is sensitive to instruction fetch
        for (int pl = pl0; pl < pl1; ++pl) {
            const DevPlane& d = a.dst[p0 + pl];
            uint32_t* o = reinterpret_cast<uint32_t*>(d.data + (long)(py0 + r0 + lr) * d.stride + gx);
            const long ostride = (long)d.stride * RPI / 2;  // words per RPI rows
            // The final output too, for a plane without restoration (DirectPlane).
            uint16_t* od = nullptr;
            int od_rows = 0;
            bool od_pair = false;
            if (DIRECT) {
                const DevPlane& D = a.direct[p0 + pl].out;
                if (D.data && gx < D.width) {
                    od = D.data + (long)(py0 + r0 + lr) * D.stride + gx;
                    od_rows = min(BH, D.height - (py0 + r0));
                    od_pair = gx + 1 < D.width;
                }
            }
#pragma unroll 1
            for (int j = j0; j < j0 + steps; ++j) {
                const uint32_t v = value(pl * plane_words + j * (RPI * PITCH / 2));
                if (col_in && lr + RPI * j < rows_here) o[j * ostride] = v;
                if (DIRECT && od && lr + RPI * j < od_rows) {
                    uint16_t* q = od + (long)j * RPI * a.direct[p0 + pl].out.stride;
                    if (od_pair) *reinterpret_cast<uint32_t*>(q) = v;
                    else *q = (uint16_t)v;
                }
            }
        }
    };
    if ((pri_on || sec_on) && active[b]) {
        const Block f = blocks[b];
        if (SHIFT) {
            auto word_tap = [&](int i) {  // i: staged index of the pair's first sample
                return (i & 1) ? s1 + ((i >> 1) - (kHalo - 2) * (PITCH / 2)) : t32 + (i >> 1);
            };
            WordTaps taps;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                taps.w[2 * k] = word_tap(base_i + f.off[k]);
                taps.w[2 * k + 1] = word_tap(base_i - f.off[k]);
            }
            rows([&](int row) { return filter_pair(cw[row], taps, row, f, pri_on, sec_on); });
        } else {
            PairTaps taps;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = base_i + (h ? -f.off[k] : f.off[k]);
                    taps.w[2 * k + h] = t32 + (i >> 1);
                    taps.sel[2 * k + h] = (i & 1) ? 0x5432u : 0x3210u;
                }
            }
            rows([&](int row) { return filter_pair(cw[row], taps, row, f, pri_on, sec_on); });
        }
    } else if (col_in) {
        rows([&](int row) { return cw[row]; });
    }
}

// A staged plane's pairs that start on odd samples, ROWS rows from row
// kHalo - 2: word w of a row holds samples 2w + 1 and 2w + 2.
template <int PITCH, int ROWS, int NT>
__device__ __forceinline__ void shift_copy(const uint16_t* t, uint32_t* shifted) {
    constexpr int WP = PITCH / 2, W0 = (kHalo - 1) / 2, NW = (PITCH - 2 * kHalo) / 2 + 1;
    const uint32_t* t32 = reinterpret_cast<const uint32_t*>(t);
    for (int i = threadIdx.x; i < ROWS * NW; i += NT) {
        const int r = i / NW, w = W0 + (i - r * NW);
        const int src = (kHalo - 2 + r) * WP + w;
        shifted[r * WP + w] = __byte_perm(t32[src], t32[src + 1], 0x5432);
    }
}

// Segment-list entry: level (6 bits) | staged offset of q0 on the segment's
// first line (13) | plane (2) | first cell of its edge (1) | last cell (1).
__device__ __forceinline__ uint32_t seg_entry(int lvl, int off, int p, bool first, bool last) {
    return (uint32_t)lvl | ((uint32_t)off << 6) | ((uint32_t)p << 19) | ((uint32_t)first << 21) |
           ((uint32_t)last << 22);
}

// The edge segments of both deblocking passes over the staged tiles of every
// plane, cell by cell.  A cell is a 4x4 block of samples at (xp, yp) =
// (px0 - 4 + 4 cc, py0 - 4 top + 4 cr), top = 2 (luma) or 1 (chroma), on
// (th/4 + 2 top) x (tw/4 + 2) cells.  Its left side is a candidate segment
// of pass 0 (vertical edges X = px0 + 4e, e <= tw/4, on rows from py0-8 or
// py0-4) and its top side one of pass 1 (horizontal edges E = py0 + 4e,
// e <= th/4, on columns from px0-4); the two share the cell's position
// checks, transform size and level word.  Each candidate gets its decision
// (7.14.2-7.14.5: on screen, transform edge, filter size, level) and joins
// its pass's list of its size class: pass 0 at s_list / s_count, pass 1 at
// s_list + kListTotal / s_count + 4.  The decisions read only the side
// information, never samples (s_count zeroed beforehand; the caller's
// barrier publishes the lists).
template <int NT>
__device__ __forceinline__ void deblock_lists(const DbCdefArgs& a, int ssx, int ssy, int x0, int y0,
                                              const SideWindow& side, uint32_t* s_list, int* s_count) {
    const int tid = threadIdx.x;
    const PlaneGeom gl = plane_geom(0, ssx, ssy), gc = plane_geom(1, ssx, ssy);
    const int nrl = gl.th / 4 + 4, ncl = gl.tw / 4 + 2;  // luma cells: rows, columns
    const int nrc = gc.th / 4 + 2, ncc = gc.tw / 4 + 2;  // chroma
    const bool u_on = a.num_planes > 1 && a.levels[2] != 0, v_on = a.num_planes > 1 && a.levels[3] != 0;
    const int n0 = nrl * ncl, n = n0 + (u_on || v_on ? nrc * ncc : 0);
    const unsigned m0 = small_div_magic(ncl), mc = small_div_magic(ncc);
    const int mi_r0 = y0 >> 2, mi_c0 = x0 >> 2;
    for (int i = tid; i < n; i += NT) {
        const bool chroma = i >= n0;
        const int j = chroma ? i - n0 : i;
        const PlaneGeom g = chroma ? gc : gl;
        const int nr = chroma ? nrc : nrl, ncol = chroma ? ncc : ncl, top = chroma ? 1 : 2;
        const int cr = small_div(j, chroma ? mc : m0), cc = j - cr * ncol;
        const DevPlane& P = a.dst[chroma ? 1 : 0];
        const int px0 = x0 >> g.sx, py0 = y0 >> g.sy;
        const int yp = py0 + 4 * (cr - top), xp = px0 - 4 + 4 * cc;
        const int col = (xp >> 2) << g.sx, row = (yp >> 2) << g.sy;
        if (!(xp >= 0 && yp >= 0 && xp < P.width && yp < P.height && col * 4 < a.coded_width &&
              row * 4 < a.coded_height))
            continue;
        const uint8_t* map = side.tx[chroma ? 1 : 0];
        const int w = (cr - top + kWinTop) * kWinCols + cc - 1 + kWinLeft;
        const int cur = map[w], cw = cur & 15, ch = cur >> 4;
        // transform edges on the cell's left (pass 0) and top (pass 1)
        const bool vert = cc >= 1 && xp > 0 && (xp & ((1 << cw) - 1)) == 0;
        const bool horz = cr >= top && cr - top <= g.th / 4 && yp > 0 && (yp & ((1 << ch) - 1)) == 0;
        if (!vert && !horz) continue;
        const int r = row | g.sy, c = col | g.sx;
        const int lw = (r - mi_r0 + kWinTop) * kWinCols + c - mi_c0 + kWinLeft;
        const uint32_t lv = a.lvl_map ? side.lvl[lw] : 0;
        const int off = (yp - py0 + kHalo) * g.pitch + (xp - px0 + kHalo);
        // Appends the edge of filter size 1 << lg to its class list, for luma
        // or for both chroma planes: level index li (7.14.5), from the cell
        // before where the cell's own level is 0.
        auto add = [&](int pass, int lg, int li, int before, bool first, bool last) {
            const int cls = lg == 2 ? 0 : chroma ? 1 : lg == 3 ? 2 : 3;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                if (v && !chroma) break;
                if (chroma && !(v ? v_on : u_on)) continue;
                int lvl;
                if (a.lvl_map) {
                    lvl = (lv >> (8 * (li + v))) & 0xFF;
                    if (lvl == 0) lvl = (side.lvl[before] >> (8 * (li + v))) & 0xFF;
                } else {
                    lvl = a.levels[li + v];
                }
                if (lvl == 0) continue;
                const int at = atomicAdd(&s_count[4 * pass + cls], 1);
                s_list[pass * kListTotal + c_list_off[cls] + at] =
                    seg_entry(lvl, off, chroma ? 1 + v : 0, first, last);
            }
        };
        if (vert) add(0, min(cw, map[w - 1] & 15), chroma ? 2 : 0, lw - (1 << g.sx), cr == 0, cr == nr - 1);
        if (horz) add(1, min(ch, map[w - kWinCols] >> 4), chroma ? 2 : 1, lw - (kWinCols << g.sy), cc == 0,
                      cc == ncol - 1);
    }
}

// The lines of one pass, filtered in one loop over its class lists laid end
// to end, so a warp changes filter code at most at a class boundary.  The
// first and last cell of an edge contribute only the lines the window needs:
// rows [py0-7, py0+th+7) / [py0-3, py0+th+3) in pass 0, columns [px0-2,
// px0+tw+2) in pass 1.  Within a pass no two edges touch a common sample, so
// the lines run in place in any order.
//
// No filter reaches past the plane: an edge of filter size n sits on a
// multiple of n (it is a transform edge of a transform at least n wide) and
// not on 0, so n samples lie before it; and the planes are Mi-padded (luma
// extents multiples of 8, chroma of 4), which leaves at least 8 samples after
// an edge of luma size 8 or 16 and 4 after any other, against reaches of 4, 7
// and, for chroma and size 4, 3.  So there are no clamped reads.  (A second,
// clamping body per class made the kernel 110 KB of code instead of 79 KB and
// a 4K 10-bit frame 1.2 % slower, without ever running.)
template <int PASS, int NT, bool HALF>
__device__ __forceinline__ void deblock_filter(const DbCdefArgs& a, int ssx, int ssy, uint16_t* smem,
                                               const uint32_t* s_list, const int* s_count,
                                               const PairStrength* s_str) {
    const int tid = threadIdx.x;
    const PlaneGeom gl = plane_geom(0, ssx, ssy), gc = plane_geom(1, ssx, ssy);
    // The lines, two per lane: lines 2h and 2h+1 of a segment (h = item & 1)
    // as the two halves of every register (filter_pair_class).  In pass 1
    // the first cell of an edge needs only its lines 2 and 3 and the last
    // only 0 and 1; pass 0 skips no pair: the lines the window does not need
    // there (line 0 of the first cell, line 3 of the last) are staged rows
    // that no later step reads, so filtering them changes nothing.
    const int c0 = s_count[0], c1 = s_count[1], c2 = s_count[2], c3 = s_count[3];
    const int pairs = 2 * (c0 + c1 + c2 + c3);
    for (int item = tid; item < pairs; item += NT) {
        int seg = item >> 1, cls = 0;
        const int h = item & 1;
        if (seg >= c0) {
            seg -= c0;
            cls = 1;
            if (seg >= c1) {
                seg -= c1;
                cls = 2;
                if (seg >= c2) {
                    seg -= c2;
                    cls = 3;
                }
            }
        }
        const uint32_t e = s_list[c_list_off[cls] + seg];
        const bool first = (e >> 21) & 1, last = (e >> 22) & 1;
        if (PASS == 1 && ((first && h == 0) || (last && h == 1))) continue;
        const int lvl = e & 63, off = (e >> 6) & 0x1FFF, p = (e >> 19) & 3;
        const int pitch = p ? gc.pitch : gl.pitch;
        uint16_t* q = smem + a.plane_off[p] + off + (PASS == 0 ? 2 * h * pitch : 2 * h);
        filter_pair_class<PASS, HALF>(cls, q, pitch, s_str[lvl], a.bit_depth - 8);
    }
    __syncthreads();
}

// The samples that vaco checks for a filtered block (decode.rs:780-841): the
// block's own luma, then, with a valid strength index, every plane's that its
// taps can reach.  Reports the first above the bit depth; the block's other
// checks have the same keys where they are made.  (Staged samples past the
// plane's borders are copies of ones inside the same reach.)
__device__ __forceinline__ void report_bad_block(const DbCdefArgs& a, int ssx, int ssy, const uint16_t* smem, int b,
                                                 int index, int mi_r0, int mi_c0) {
    const int by = b >> 3, bx = b & 7;
    const unsigned long long pos = ((unsigned long long)(mi_r0 + 2 * by) * a.mi_cols + mi_c0 + 2 * bx) * 4;
#pragma unroll 1
    for (int k = 0; k <= (index < 8 ? a.num_planes : 0); ++k) {  // luma alone, then the planes with their reach
        const PlaneGeom g = plane_geom(k > 1 ? 1 : 0, ssx, ssy);
        const int bw = 8 >> g.sx, bh = 8 >> g.sy, reach = k ? 2 : 0;
        const uint16_t* t =
            smem + a.plane_off[max(k - 1, 0)] + (kHalo + by * bh - reach) * g.pitch + kHalo + bx * bw - reach;
        int most = 0;
#pragma unroll 1
        for (int i = 0; i < (bh + 2 * reach) * (bw + 2 * reach); ++i)
            most = max(most, (int)t[i / (bw + 2 * reach) * g.pitch + i % (bw + 2 * reach)]);
        if (most >> a.bit_depth) {
            report_error(a.status, STAGE_CDEF, pos + k, k ? VACO_AV1_MSG_CDEF_BLOCK_PARAMS : VACO_AV1_MSG_CDEF_SAMPLE);
            return;
        }
    }
}

// One 64x64 filter block (tile_x, tile_y) of one frame.  Every thread of the
// CTA calls it; it ends with all threads past their last shared-memory use
// only after the caller's next __syncthreads().
// ALONE: the call may be cdef_picture's, for CDEF alone, which has no transform
// sizes.
template <int NT, int LAYOUT, class Block, bool DIRECT, bool ALONE>
__device__ __forceinline__ void dbcdef_tile(const DbCdefArgs& a, int tile_x, int tile_y) {
    constexpr int kWarpsNT = NT / 32;
    constexpr bool kHalf = std::is_same<Block, HalfBlock>::value;  // samples of up to 10 bits
    // chroma subsampling: LAYOUT = ssx | ssy << 1 fixes it at compile time
    // (every plane geometry below becomes a constant); LAYOUT < 0 reads it
    const int ssx = LAYOUT < 0 ? a.ssx : (LAYOUT & 1), ssy = LAYOUT < 0 ? a.ssy : (LAYOUT >> 1);
    extern __shared__ __align__(16) uint16_t smem[];
    __shared__ uint32_t s_cost[8][64];  // per direction and block
    __shared__ Block s_block[2][64];  // luma, chroma (U and V share strengths and directions)
    __shared__ uint8_t s_active[64];
    __shared__ int s_count[8];  // list lengths per size class, pass 0 then pass 1
    __shared__ PairStrength s_str[64];  // per loop-filter level, for this frame's sharpness and depth
    // The deblocking lists and side window are dead once deblocking is done;
    // the CDEF phase reuses their space for the odd-aligned luma pairs.
    __shared__ union {
        struct {
            uint32_t list[2 * kListTotal];  // per pass and size class, see seg_entry()
            SideWindow side;
        } db;
        uint32_t shifted[kShiftWords];
    } s_u;
    uint32_t* s_list = s_u.db.list;
    SideWindow& s_side = s_u.db.side;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mi_r0 = tile_y * 16, mi_c0 = tile_x * 16;
    const int x0 = mi_c0 * 4, y0 = mi_r0 * 4;

    // ---- CDEF block activity (decode.rs:772-779)
    const long slot = (long)(mi_r0 >> 4) * a.cdef_stride + (mi_c0 >> 4);
    const int index = (a.cdef_on && slot < a.cdef_count) ? __ldg(a.cdef_idx + slot) : -1;
    bool act = false;
    if (tid < 64) {
        const int r = mi_r0 + (tid >> 3) * 2, c = mi_c0 + (tid & 7) * 2;
        if (r < a.mi_rows && c < a.mi_cols && index >= 0) {
            auto sk = [&](int rr, int cc) {
                return rr < a.mi_rows && cc < a.mi_cols && a.skip[(long)rr * a.mi_cols + cc] != 0;
            };
            act = !(sk(r, c) && sk(r + 1, c) && sk(r, c + 1) && sk(r + 1, c + 1));
        }
        s_active[tid] = act;
    }

    // the deblocking lists' lengths and strengths, published by the staging
    // barrier below
    if (tid < 8) s_count[tid] = 0;
    if (a.deblock_on && tid < 64) s_str[tid] = pair_strength<kHalf>(strength_of(tid, a.sharpness), a.bit_depth - 8);

    // ---- every plane's tile with an 8-sample halo (edge-clamped).  Whole
    // 16-byte chunks inside the plane go by cp.async, all in flight at once;
    // chunks that straddle the left/right plane edge are gathered sample by
    // sample.  Rows past the top/bottom edge repeat the edge row.  (Staging
    // interior tiles with 2-D tensor copies instead measured 1.4 % slower
    // for the whole chain: the extra path costs more than the copies save.)
    // A tile whose halo lies inside every plane (nine in ten of a 4K frame)
    // steps down its columns by pointer increments alone.
    auto inside = [&](int p) {
        const PlaneGeom g = plane_geom(p, ssx, ssy);
        const int px0 = x0 >> g.sx, py0 = y0 >> g.sy;
        return px0 >= kHalo && py0 >= kHalo && px0 + g.tw + kHalo <= a.src[p].width &&
               py0 + g.th + kHalo <= a.src[p].height;
    };
    const bool interior = a.vec_ok && inside(0) && (a.num_planes == 1 || inside(1));
    for (int p = 0; p < a.num_planes; ++p) {
        const PlaneGeom g = plane_geom(p, ssx, ssy);
        const DevPlaneC& P = a.src[p];
        uint16_t* t = smem + a.plane_off[p];
        const int px0 = x0 >> g.sx, py0 = y0 >> g.sy;
        const int vpr = g.pitch / 8;
        if (interior) {
            const int step = NT / vpr, r0 = tid / vpr, cv = tid - r0 * vpr;  // vpr is 10 or 6
            if (r0 >= step) continue;
            const uint16_t* src = P.data + (long)(py0 - kHalo + r0) * P.stride + px0 - kHalo + cv * 8;
            unsigned dst = (unsigned)__cvta_generic_to_shared(t + r0 * g.pitch + cv * 8);
            const long src_step = (long)step * P.stride;
            for (int r = r0; r < g.rows; r += step) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
                src += src_step;
                dst += (unsigned)(step * g.pitch * 2);
            }
            continue;
        }
        const unsigned mv = small_div_magic(vpr);
        for (int v = tid; v < g.rows * vpr; v += NT) {
            const int r = small_div(v, mv), cv = v - r * vpr;
            const int y = clampi(py0 - kHalo + r, 0, P.height - 1);
            const int x = px0 - kHalo + cv * 8;
            const uint16_t* row = P.data + (long)y * P.stride;
            uint16_t* d = t + r * g.pitch + cv * 8;
            if (a.vec_ok && x >= 0 && x + 8 <= P.width) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(d);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(row + x) : "memory");
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) d[k] = __ldg(row + clampi(x + k, 0, P.width - 1));
            }
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");

    // ---- the side information the deblocking decisions read, while the
    // copies are in flight (cells the two passes touch; see SideWindow).  Each
    // cell is checked where it is loaded: the windows of all tiles together
    // hold exactly the maps' cells.
    if (!ALONE || a.tx_luma) {
        const int crows = (a.mi_rows + ssy) >> ssy, ccols = (a.mi_cols + ssx) >> ssx;
        const int cr0 = (mi_r0 >> ssy) - kWinTop, cc0 = (mi_c0 >> ssx) - kWinLeft;
        int bad = 0;
        for (int i = tid; i < kWinCells; i += NT) {
            const int wr = i / kWinCols, wc = i - wr * kWinCols;
            const int r = mi_r0 - kWinTop + wr, c = mi_c0 - kWinLeft + wc;
            if (r >= 0 && c >= 0 && r < a.mi_rows && c < a.mi_cols) {
                const long cell = (long)r * a.mi_cols + c;
                const int t = __ldg(a.tx_luma + cell);
                s_side.tx[0][i] = tx_logs(t);
                bad |= t > 18;
                if (a.lvl_map) {
                    const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(a.lvl_map) + cell);
                    // A level above 63 is reported and cut: list entries
                    // hold 6 bits of it beside the segment's offset.
                    s_side.lvl[i] = v & 0x3F3F3F3Fu;
                    bad |= (v & 0xC0C0C0C0u) != 0;
                }
            }
            if (a.num_planes > 1 && cr0 + wr >= 0 && cc0 + wc >= 0 && cr0 + wr < crows && cc0 + wc < ccols) {
                const int t = __ldg(a.tx_chroma + (long)(cr0 + wr) * ccols + cc0 + wc);
                s_side.tx[1][i] = tx_logs(t);
                bad |= t > 18;
            }
        }
        if (bad) report_error(a.status, STAGE_DEBLOCK, 0, VACO_AV1_MSG_DB_PARAMS);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    const bool any_active = __syncthreads_or(act);

    // ---- input check from shared memory
    // Every staged sample, halo included: the halo holds samples of the
    // same planes (edge-clamped copies past their borders), so the tiles
    // together check exactly the planes' samples, and a flat pass over
    // the staged vectors needs no per-row indexing.
    {
        const uint32_t hi = ((0xFFFFu << a.bit_depth) & 0xFFFFu) * 0x10001u;  // bits above the depth, per lane
        const uint4* v = reinterpret_cast<const uint4*>(smem);
        uint32_t acc = 0;
        for (int i = tid; i < a.staged_vectors; i += NT) {
            const uint4 w = v[i];
            acc |= w.x | w.y | w.z | w.w;
        }
        // A report a warp: one a thread, all to one word, took a 4K frame of
        // bad samples alone from 161 to 431 us.
        if (__any_sync(0xFFFFFFFFu, (acc & hi) != 0) && lane == 0) {
            if (ALONE && !a.tx_luma) s_count[0] = 1;  // without deblocking nothing else counts there
            else report_error(a.status, STAGE_DEBLOCK, 1, VACO_AV1_MSG_DB_SAMPLE);
        }
    }

    // ---- deblocking, pass 0 (vertical edges) then pass 1 (horizontal edges)
    if (a.deblock_on) {
        deblock_lists<NT>(a, ssx, ssy, x0, y0, s_side, s_list, s_count);
        __syncthreads();
        deblock_filter<0, NT, kHalf>(a, ssx, ssy, smem, s_list, s_count, s_str);
        deblock_filter<1, NT, kHalf>(a, ssx, ssy, smem, s_list + kListTotal, s_count + 4, s_str);
    } else {
        // the sample check above reads every staged sample, the sentinel
        // phase below overwrites some
        __syncthreads();
        if (ALONE && !a.tx_luma && s_count[0]) {  // a bad sample: apply_cdef's rule
            if (tid < 64 && s_active[tid]) report_bad_block(a, ssx, ssy, smem, tid, index, mi_r0, mi_c0);
            __syncthreads();
        }
    }

    // ---- stripe-boundary rows of the deblocked picture for restoration: rows
    // y with (y + offset + 2) mod stripe < 4, stored at 4*boundary + that
    // remainder (boundary = (y + offset + 2) / stripe >= 1).  A tile is one
    // stripe high, so it holds the four rows around its own boundary, from row
    // th - offset - 2 on: 8-sample vectors, one a thread (64 for 4:2:0).  The
    // compact buffers' rows are padded to 64 samples, which takes the vector
    // that a 4:2:0 chroma plane's last columns share with the padding.
    {
        constexpr int nl = 64 / 8, kMost = 3 * nl;  // vectors of a row: luma's, all planes' at most
        const int ncv = a.num_planes > 1 ? (64 >> ssx) / 8 : 0;
        const int sub_row = tid / kMost, i = tid - sub_row * kMost;
        if (tid < 4 * kMost && i < nl + 2 * ncv) {
            const int p = i < nl ? 0 : i < nl + ncv ? 1 : 2;
            const int c = 8 * (i - (p == 0 ? 0 : nl + (p - 1) * ncv));
            const DevPlane& R = a.pre_rows[p];
            const PlaneGeom g = plane_geom(p ? 1 : 0, ssx, ssy);
            const int off = 8 >> g.sy, px0 = x0 >> g.sx, py0 = y0 >> g.sy;
            const int r = g.th - off - 2 + sub_row;
            if (R.data && px0 + c < a.dst[p].width && py0 + r < a.dst[p].height)
                *reinterpret_cast<uint4*>(R.data + (long)(4 * (py0 / g.th + 1) + sub_row) * R.stride + px0 + c) =
                    *reinterpret_cast<const uint4*>(smem + a.plane_off[p] + (r + kHalo) * g.pitch + kHalo + c);
        }
    }

    // ---- CDEF on the deblocked tile
    if (!any_active) {
        // Nothing filtered (or CDEF off): the output is the deblocked tile.
        for (int p = 0; p < a.num_planes; ++p) {
            const PlaneGeom g = plane_geom(p, ssx, ssy);
            const DevPlane& d = a.dst[p];
            const int px0 = x0 >> g.sx, py0 = y0 >> g.sy;
            const DirectPlane* D = DIRECT ? &a.direct[p] : nullptr;
            const uint16_t* t = smem + a.plane_off[p];
            if (a.dst_vec && !(D && D->out.data) && px0 + g.tw <= d.width) {  // whole rows of 16-byte vectors
                const int lv = 3 - g.sx;  // log2 of the vectors of a row
                for (int i = tid; i < g.th << lv; i += NT) {
                    const int r = i >> lv, c = (i & ((1 << lv) - 1)) * 8, y = py0 + r;
                    if (y >= d.height) break;
                    *reinterpret_cast<uint4*>(d.data + (long)y * d.stride + px0 + c) =
                        *reinterpret_cast<const uint4*>(t + (r + kHalo) * g.pitch + kHalo + c);
                }
                continue;
            }
            for (int r = warp; r < g.th; r += kWarpsNT) {
                const int y = py0 + r;
                if (y >= d.height) break;
                for (int c = lane; c < g.tw; c += 32) {
                    const int x = px0 + c;
                    if (x >= d.width) continue;
                    const uint16_t v = t[(r + kHalo) * g.pitch + c + kHalo];
                    d.data[(long)y * d.stride + x] = v;
                    // the final output too, for a plane without restoration
                    if (D && D->out.data && y < D->out.height && x < D->out.width)
                        D->out.data[(long)y * D->out.stride + x] = v;
                }
            }
        }
        return;
    }
    // Samples outside the plane become the "unavailable" sentinel for CDEF.
    for (int p = 0; p < a.num_planes; ++p) {
        const PlaneGeom g = plane_geom(p, ssx, ssy);
        const DevPlane& d = a.dst[p];
        const int px0 = x0 >> g.sx, py0 = y0 >> g.sy;
        if (px0 + g.tw + 2 <= d.width && py0 + g.th + 2 <= d.height && px0 >= 2 && py0 >= 2) continue;
        uint16_t* t = smem + a.plane_off[p];
        const int wr = g.th + 4, wc = g.tw + 4;
        const unsigned mw = small_div_magic(wc);
        for (int i = tid; i < wr * wc; i += NT) {
            const int r = small_div(i, mw), c = i - r * wc;
            const int y = py0 - 2 + r, x = px0 - 2 + c;
            if (y < 0 || x < 0 || y >= d.height || x >= d.width)
                t[(r + kHalo - 2) * g.pitch + (c + kHalo - 2)] = (uint16_t)kSent;
        }
    }
    __syncthreads();

    // The CDEF windows' pairs that start on odd samples (rows kHalo-2 ..
    // kHalo+th+1, first samples on columns kHalo-1 .. kHalo+tw-1), as words
    // on the staged row pitch, so the pair filter reads every tap with one
    // aligned load: luma, and 4:2:0 chroma, whose copies lie as far apart as
    // the staged planes (the other layouts' do not fit beside luma's).
    shift_copy<64 + 2 * kHalo, kShiftRows, NT>(smem + a.plane_off[0], s_u.shifted);
    if (a.num_planes > 1 && ssx == 1 && ssy == 1) {
        uint32_t* sc = s_u.shifted + kShiftRows * (64 + 2 * kHalo) / 2;
        shift_copy<32 + 2 * kHalo, 32 + 4, NT>(smem + a.plane_off[1], sc);
        shift_copy<32 + 2 * kHalo, 32 + 4, NT>(smem + a.plane_off[2], sc + (32 + 2 * kHalo) * (32 + 2 * kHalo) / 2);
    }

    // Direction search: a warp takes 32 blocks, one per lane, and a direction
    // pair (d, d + 4), or with 16 warps and more one direction, so every
    // branch below is warp-uniform.
    const int lpitch = 64 + 2 * kHalo;
    constexpr int kDirJobs = kWarpsNT > 8 ? 16 : 8;
    for (int job = warp; job < kDirJobs; job += kWarpsNT) {
        const int pair = job & 3, b = (((job >> 2) & 1) << 5) + lane;
        if (s_active[b]) {
            const uint16_t* blk = smem + a.plane_off[0] + (kHalo + (b >> 3) * 8) * lpitch + kHalo + (b & 7) * 8;
            if (kDirJobs == 16) {
                const int d = pair + ((job >> 3) << 2);
                s_cost[d][b] = dir_cost_of(d, blk, lpitch, a.shift);
            } else {
                uint32_t lo, hi;
                dir_costs_pair(pair, blk, lpitch, a.shift, lo, hi);
                s_cost[pair][b] = lo;
                s_cost[pair + 4][b] = hi;
            }
        }
    }
    __syncthreads();
    // Per block, luma and chroma (one thread each): direction, strengths, checks.
    for (int i = tid; i < (a.num_planes > 1 ? 128 : 64); i += NT) {
        if (!s_active[i & 63]) continue;
        const int b = i & 63;
        const bool chroma = i >= 64;
        int dir;
        uint32_t var;
        best_direction(s_cost, b, dir, var);
        int sp = 0, ss = 0;
        if (index < 8) {
            sp = chroma ? a.uv_pri[index] : a.y_pri[index];
            ss = chroma ? a.uv_sec[index] : a.y_sec[index];
        }
        int primary = (sp << a.shift) & 0xFFFF;
        const int secondary = (ss << a.shift) & 0xFFFF;
        const int chosen = primary == 0 ? 0 : chroma ? chroma_direction(dir, ssx, ssy) : dir;
        if (!chroma) primary = adjust_strength(primary, var);
        const int damping = (a.damping + a.shift - (chroma ? 1 : 0)) & 0xFF;
        // Luma and chroma report their own failures; the status word keeps the
        // lowest (block, plane) key, i.e. the first plane vaco would reject
        // (V, whose parameters are U's, never comes first).
        if (index >= 8 || damping > 12 || primary > (15 << a.shift) || secondary > (4 << a.shift)) {
            const int r = mi_r0 + (b >> 3) * 2, c = mi_c0 + (b & 7) * 2;
            report_error(a.status, STAGE_CDEF, ((unsigned long long)r * a.mi_cols + c) * 4 + 1 + (chroma ? 1 : 0),
                         index >= 8 ? VACO_AV1_MSG_CDEF_STRENGTH_INDEX : VACO_AV1_MSG_CDEF_BLOCK_PARAMS);
        }
        const int pitch = plane_geom(chroma ? 1 : 0, ssx, ssy).pitch;
        make_block(s_block[chroma ? 1 : 0][b], chosen, primary, secondary, min(damping, 12), a.shift, pitch);
    }
    __syncthreads();

    // Filtering: pixel pairs (two 16-bit lanes per register), one warp per
    // block row, lanes across the tile width; luma, then both chroma planes.
    // Tap sets of the tile's preset (uniform over the tile).
    const bool y_pri_on = index >= 8 || a.y_pri[index] != 0, y_sec_on = index >= 8 || a.y_sec[index] != 0;
    constexpr int kParts = kWarpsNT > 8 ? kWarpsNT / 8 : 1;  // warps per block row
    const int row0 = warp / kParts, part = warp % kParts;
    constexpr int kRowStep = kWarpsNT / kParts;
    for (int br = row0; br < 8; br += kRowStep)
        filter_block_row<64 + 2 * kHalo, 8, 1, 1, kParts, true, DIRECT>(a, 0, smem + a.plane_off[0], s_u.shifted, 0,
                                                                        x0, y0, s_active, s_block[0], y_pri_on,
                                                                        y_sec_on, br, part, lane, 0);
    if (a.num_planes > 1) {
        const bool c_pri_on = index >= 8 || a.uv_pri[index] != 0, c_sec_on = index >= 8 || a.uv_sec[index] != 0;
        const uint16_t* tc = smem + a.plane_off[1];
        const int plane_words = (int)(a.plane_off[2] - a.plane_off[1]) / 2;
        const int px0 = x0 >> ssx, py0 = y0 >> ssy;
        // tile layouts: 64x64 (4:4:4), 32x32 (4:2:0), 32x64 (4:2:2)
        for (int br = row0; br < 8; br += kRowStep) {
            if (ssx == 0)
                filter_block_row<64 + 2 * kHalo, 8, 1, 2, kParts, false, DIRECT>(
                    a, 1, tc, nullptr, plane_words, px0, py0, s_active, s_block[1], c_pri_on, c_sec_on, br, part, lane,
                    ssx);
            else if (ssy == 1)
                filter_block_row<32 + 2 * kHalo, 4, 2, 2, kParts, true, DIRECT>(
                    a, 1, tc, s_u.shifted + kShiftRows * (64 + 2 * kHalo) / 2, plane_words, px0, py0, s_active,
                    s_block[1], c_pri_on, c_sec_on, br, part, lane, ssx);
            else
                filter_block_row<32 + 2 * kHalo, 8, 2, 2, kParts, false, DIRECT>(
                    a, 1, tc, nullptr, plane_words, px0, py0, s_active, s_block[1], c_pri_on, c_sec_on, br, part, lane,
                    ssx);
        }
    }
}

// NT threads per tile, MIN_CTAS CTAs per SM.  The per-frame path runs 512
// threads at 2 CTAs per SM for frames of up to two tiles per SM (see
// launch_dbcdef_as()), else 256 threads at 4 CTAs per SM (64 registers a
// thread), measured at least as fast as 3 (80 registers) on 1080p and on 2560-,
// 2880- and 3840-wide frames (1.5-2 % faster on the last two); 128 threads at 5
// CTAs per SM is the smaller-CTA shape (shorter barriers, about the same warps
// per SM), which only the tuning selects: 13 % slower on the mix of frames
// (3.37 against 2.97 ms for 64 frames), 15 % on a 4K frame (0.152, 0.132 ms).
// DIRECT: a body that also writes the output of planes without restoration
// (DirectPlane); the code for it measured 3 % slower on frames that have no
// such plane, so it is a separate body.
template <int NT, int MIN_CTAS, int LAYOUT, class Block, bool DIRECT = false>
__global__ void __launch_bounds__(NT, MIN_CTAS) dbcdef_kernel(DbCdefArgs a) {
    overlap_prologue();
    dbcdef_tile<NT, LAYOUT, Block, DIRECT, !DIRECT>(a, blockIdx.x, a.tile_row0 + blockIdx.y);
}

// Batched form: one CTA per tile of all frames of a batch, frames laid end to
// end in `tile_prefix` order, so frames of any size share one launch and the
// hardware hands out the tiles in that order.  MIN_CTAS as for dbcdef_kernel.
// (A persistent form, CTAs taking tiles from a device queue, kept its loop
// state and the frame record live across the tile and spilled registers: it
// measured 4 % slower on 4K frames.)  LAYOUT as for dbcdef_tile: a batch
// whose frames share one chroma layout takes the body compiled for it.
template <int NT, int MIN_CTAS, int LAYOUT, class Block>
__global__ void __launch_bounds__(NT, MIN_CTAS) dbcdef_batch_kernel(const DbCdefArgs* __restrict__ frames,
                                                                    const int* __restrict__ tile_prefix, int n) {
    overlap_prologue();
    const int f = frame_of_tile(tile_prefix, n, blockIdx.x);
    const DbCdefArgs& a = frames[f];
    const int local = blockIdx.x - tile_prefix[f];
    const int tiles_x = (a.mi_cols + 15) / 16;
    dbcdef_tile<NT, LAYOUT, Block, false, false>(a, local % tiles_x, local / tiles_x);
}

}  // namespace

size_t dbcdef_args_size() { return sizeof(DbCdefArgs); }

// Kernel arguments of one frame; returns the dynamic shared memory it needs.
size_t build_dbcdef_args(const DbCdefLaunch& L, void* out) {
    DbCdefArgs a;
    memset(&a, 0, sizeof a);
    const int np = L.info.monochrome ? 1 : 3;
    bool vec = true, dst_vec = true;
    size_t off = 0;
    for (int p = 0; p < 3; ++p) {
        a.src[p] = DevPlaneC{L.src.planes[p], L.src.width[p], L.src.height[p], L.src.stride[p]};
        a.dst[p] = DevPlane{L.dst.planes[p], L.dst.width[p], L.dst.height[p], L.dst.stride[p]};
        a.pre_rows[p] = L.pre_rows[p];
        a.plane_off[p] = off;
        if (p < np) {
            vec = vec && (L.src.stride[p] % 8 == 0) && ((uintptr_t)L.src.planes[p] % 16 == 0);
            dst_vec = dst_vec && (L.dst.stride[p] % 8 == 0) && ((uintptr_t)L.dst.planes[p] % 16 == 0);
            const int sx = p ? L.info.subsampling_x : 0, sy = p ? L.info.subsampling_y : 0;
            off += (size_t)((64 >> sx) + 2 * kHalo) * ((64 >> sy) + 2 * kHalo);
        }
    }
    a.num_planes = np;
    a.ssx = np > 1 ? L.info.subsampling_x : 0;
    a.ssy = np > 1 ? L.info.subsampling_y : 0;
    a.bit_depth = L.info.bit_depth;
    a.shift = L.info.bit_depth - 8;
    a.mi_rows = L.info.mi_rows;
    a.mi_cols = L.info.mi_cols;
    a.coded_width = L.info.coded_width;
    a.coded_height = L.info.coded_height;
    a.tx_luma = L.tx_luma;
    a.tx_chroma = L.tx_chroma;
    a.lvl_map = L.lvl_map;
    for (int k = 0; k < 4; ++k) a.levels[k] = L.deblock.levels[k];
    a.sharpness = L.deblock.sharpness;
    a.deblock_on = !(L.deblock.levels[0] == 0 && L.deblock.levels[1] == 0);
    bool all_zero = true;
    for (int k = 0; k < 8; ++k)
        all_zero = all_zero && L.cdef.y_primary[k] == 0 && L.cdef.y_secondary[k] == 0 && L.cdef.uv_primary[k] == 0 &&
                   L.cdef.uv_secondary[k] == 0;
    a.cdef_on = L.cdef.enabled && !all_zero && L.skip != nullptr;
    a.skip = L.skip;
    a.cdef_idx = L.cdef_idx;
    a.cdef_stride = L.cdef_stride;
    a.cdef_count = L.cdef_idx ? L.cdef_count : 0;
    a.damping = L.cdef.damping;
    for (int k = 0; k < 8; ++k) {
        a.y_pri[k] = L.cdef.y_primary[k];
        a.y_sec[k] = L.cdef.y_secondary[k];
        a.uv_pri[k] = L.cdef.uv_primary[k];
        a.uv_sec[k] = L.cdef.uv_secondary[k];
    }
    a.status = L.status;
    a.vec_ok = vec;
    a.dst_vec = dst_vec;
    a.tile_row0 = L.tile_row0;
    a.staged_vectors = (int)(off / 8);  // each staged plane is a multiple of 8 samples
    for (int p = 0; p < 3; ++p) a.direct[p] = p < np ? L.direct[p] : DirectPlane{};
    memcpy(out, &a, sizeof a);
    return off * sizeof(uint16_t);
}

// Per-device cache, shared by every host thread that launches: an atomic, so
// concurrent first launches on a device only repeat idempotent set-up.
std::atomic<unsigned long long> g_attr_devices{0};

cudaError_t dbcdef_kernel_attributes() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !(g_attr_devices.load(std::memory_order_acquire) & (1ull << dev))) {
        constexpr int kMaxSmem = 96 * 1024;
        const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
        cudaError_t e = cudaSuccess;
        auto optin = [&](auto block) {
            using B = decltype(block);
            for (auto k : {dbcdef_kernel<256, 4, 0, B>, dbcdef_kernel<256, 4, 1, B>, dbcdef_kernel<256, 4, 3, B>,
                           dbcdef_kernel<256, 4, 0, B, true>, dbcdef_kernel<256, 4, 1, B, true>,
                           dbcdef_kernel<256, 4, 3, B, true>, dbcdef_kernel<128, 5, 0, B>, dbcdef_kernel<128, 5, 1, B>,
                           dbcdef_kernel<128, 5, 3, B>, dbcdef_kernel<512, 2, 0, B>, dbcdef_kernel<512, 2, 1, B>,
                           dbcdef_kernel<512, 2, 3, B>, dbcdef_kernel<512, 2, 0, B, true>,
                           dbcdef_kernel<512, 2, 1, B, true>, dbcdef_kernel<512, 2, 3, B, true>})
                if (e == cudaSuccess) e = cudaFuncSetAttribute(k, attr, kMaxSmem);
            for (auto k : {dbcdef_batch_kernel<256, 4, 0, B>, dbcdef_batch_kernel<256, 4, 1, B>,
                           dbcdef_batch_kernel<256, 4, 3, B>, dbcdef_batch_kernel<256, 4, -1, B>,
                           dbcdef_batch_kernel<128, 5, -1, B>})
                if (e == cudaSuccess) e = cudaFuncSetAttribute(k, attr, kMaxSmem);
        };
        optin(HalfBlock{});
        optin(PairBlock{});
        if (e != cudaSuccess) return e;
        g_attr_devices.fetch_or(1ull << dev, std::memory_order_release);
    }
    return cudaSuccess;
}

// One kernel per chroma layout (4:4:4 and monochrome, 4:2:2, 4:2:0) and block
// form (half-precision CDEF taps up to 10 bits, integer ones above); a frame
// with a plane written straight to the output takes a body that does so.
template <int NT, int MIN_CTAS, class Block, bool DIRECT>
static cudaError_t launch_dbcdef_nt(const DbCdefArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    const int layout = a.ssx | a.ssy << 1;
    auto k = layout == 3   ? dbcdef_kernel<NT, MIN_CTAS, 3, Block, DIRECT>
             : layout == 1 ? dbcdef_kernel<NT, MIN_CTAS, 1, Block, DIRECT>
                           : dbcdef_kernel<NT, MIN_CTAS, 0, Block, DIRECT>;
    return launch_overlapped(k, grid, dim3(NT), smem, stream, a);
}

template <class Block>
static cudaError_t launch_dbcdef_as(const DbCdefArgs& a, bool direct, int threads, int sm_count, dim3 grid,
                                    size_t smem, cudaStream_t stream) {
    // A frame whose tiles are all resident at 512 threads each (two CTAs per
    // SM) takes one tile's latency, which the second set of warps shortens:
    // 640x360 23.0 -> 18.2 us, 1280x720 26.1 -> 23.6 us.  With more tiles than
    // that a CTA per SM more is the better use of the registers: 1440x810
    // (299 tiles) 27.5 us at 256 threads, 31.5 at 512.  (1024 threads, one CTA
    // per SM: 17.7 us at 640x360, 30.0 at 1280x720.)
    if (threads != 128 && (long)grid.x * grid.y <= 2L * sm_count)
        return direct ? launch_dbcdef_nt<512, 2, Block, true>(a, grid, smem, stream)
                      : launch_dbcdef_nt<512, 2, Block, false>(a, grid, smem, stream);
    if (direct) return launch_dbcdef_nt<256, 4, Block, true>(a, grid, smem, stream);
    if (threads == 128) return launch_dbcdef_nt<128, 5, Block, false>(a, grid, smem, stream);
    return launch_dbcdef_nt<256, 4, Block, false>(a, grid, smem, stream);
}

cudaError_t launch_dbcdef(const DbCdefLaunch& L, cudaStream_t stream) {
    DbCdefArgs a;
    const size_t smem = build_dbcdef_args(L, &a);
    cudaError_t e = dbcdef_kernel_attributes();
    if (e != cudaSuccess) return e;
    const int tile_rows = L.tile_rows < 0 ? div_up(L.info.mi_rows, 16) - L.tile_row0 : L.tile_rows;
    if (tile_rows <= 0) return cudaSuccess;
    const dim3 grid(div_up(L.info.mi_cols, 16), tile_rows);
    const bool direct = a.direct[0].out.data || a.direct[1].out.data || a.direct[2].out.data;
    return a.bit_depth <= 10 ? launch_dbcdef_as<HalfBlock>(a, direct, L.threads, L.sm_count, grid, smem, stream)
                             : launch_dbcdef_as<PairBlock>(a, direct, L.threads, L.sm_count, grid, smem, stream);
}

template <class Block>
static cudaError_t launch_dbcdef_batch_as(const DbCdefArgs* args, const int* dev_prefix, int n, int tiles, size_t smem,
                                          int threads, int layout, cudaStream_t stream) {
    using K = void (*)(const DbCdefArgs*, const int*, int);
    K k;
    if (threads == 128) {
        k = dbcdef_batch_kernel<128, 5, -1, Block>;
    } else {  // as the per-frame kernel; at 3 CTAs per SM (80 registers) the mix of frames is 4.5 % slower
        k = layout == 3 ? dbcdef_batch_kernel<256, 4, 3, Block> : layout == 1 ? dbcdef_batch_kernel<256, 4, 1, Block>
          : layout == 0 ? dbcdef_batch_kernel<256, 4, 0, Block> : dbcdef_batch_kernel<256, 4, -1, Block>;
    }
    return launch_overlapped(k, dim3(tiles), dim3(threads == 128 ? 128 : 256), smem, stream, args, dev_prefix, n);
}

cudaError_t launch_dbcdef_batch(const void* dev_args, const int* dev_prefix, int n, int tiles, size_t smem,
                                int threads, int layout, int max_bit_depth, cudaStream_t stream) {
    if (tiles <= 0) return cudaSuccess;
    cudaError_t e = dbcdef_kernel_attributes();
    if (e != cudaSuccess) return e;
    const DbCdefArgs* args = static_cast<const DbCdefArgs*>(dev_args);
    return max_bit_depth <= 10
               ? launch_dbcdef_batch_as<HalfBlock>(args, dev_prefix, n, tiles, smem, threads, layout, stream)
               : launch_dbcdef_batch_as<PairBlock>(args, dev_prefix, n, tiles, smem, threads, layout, stream);
}

}  // namespace vaco
