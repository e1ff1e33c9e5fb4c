// Device side of the exact diagram (exact.cu), shared by the single-image and
// the batched pipelines (an image is one padded canvas of the atlas; a single
// image is the whole plane).
//
// Column pass: each cell's signed row offset to the nearest seed of its own
// column (ties to the lower one, the higher id), two bytes per cell, and a
// table that turns (column, row of a seed) into the seed's id.
// Row pass: each cell's winner among its row's column candidates, and its id.
#pragma once

#include "common.cuh"

namespace idl {

struct XImg {
    int ox, oy, Wp, Hp;    // padded canvas origin and size on the plane
    int pair_off;          // first entry of this image in the column-pair table
    int row_off;           // first entry in the row table
    int band_off;          // first entry in the band table
    int s0, s1;            // its seeds: ids [s0, s1), (x, y)-sorted
    int P;                 // padding around the image proper
    long long bit0;        // its first occupancy bit (column-major over the image proper)
};

constexpr int BAND = 64;                       // rows a thread of the column pass walks
constexpr int16_t NO_SEED = (int16_t)-32768;   // a column without seeds

__host__ __device__ inline int x_bands(const XImg& m) { return (m.Hp + BAND - 1) / BAND; }

// The seeds' occupancy bits, column-major image after image, and the number of
// seeds before each word (seeds.cu): a seed's rank is the number before its bit.
struct SeedRanks {
    const uint32_t* bits;
    const int32_t* before;
    const int32_t* label;   // label of each rank, ties going to the higher label; null: the rank itself
};

// Per band of rows and column: its seeds in the band as a 64-bit mask of the
// rows (z, w) and the rank of the first of them (x).
struct SeedBands {
    const uint4* band;
    const int32_t* label;   // as in SeedRanks
};

// Rank of the seed at (x, y) of the plane, which must exist.  One load however
// dense the seeds: a walk along the column's seeds from the band's first one
// took ten loads in a row per cell at one seed in three cells (row pass of
// 2048 x 2048: 291 us, now 88; at 200 000 seeds in 4096 x 4096 134 and 130
// us), and the occupancy bits and their ranks, two loads from column-major
// tables, 147 us there.
__device__ __forceinline__ int32_t x_seed_at(const SeedBands& B, const XImg& m, int x, int y)
{
    const unsigned row = (unsigned)(y - m.oy), k = row % BAND;
    const uint4 e = __ldg(&B.band[m.band_off + (int)(row / BAND) * m.Wp + (x - m.ox)]);
    const uint32_t low = k < 32 ? (1u << k) - 1u : 0xFFFFFFFFu, high = k > 32 ? (1u << (k - 32)) - 1u : 0u;
    return (int32_t)e.x + __popc(e.z & low) + __popc(e.w & high);
}

// One thread walks two adjacent columns (the pair starting at image column c)
// through the rows of one band, so that a warp writes 128 bytes of a row at
// once.  The band's seeds of a column come as a 64-bit mask from the occupancy
// bits, the seeds before and after the band by their ranks: the walk itself
// loads nothing (dense columns: 24 us instead of 44 at 2048 x 2048, one seed in
// three cells).  Two bytes per cell and a table entry per 64 are written.
__device__ __forceinline__ void x_column_pair(const uint32_t* __restrict__ pos, const SeedRanks& ranks,
                                              const XImg& m, int c, int band,
                                              int pitch, int16_t* __restrict__ off, uint4* __restrict__ bands)
{
    static_assert(BAND == 64, "a column's rows of a band are the bits of one 64-bit mask");
    const int y0 = band * BAND, y1 = min(m.Hp, y0 + BAND);
    const int W = m.Wp - 2 * m.P, H = m.Hp - 2 * m.P;
    const int r0 = min(max(y0 - m.P, 0), H), r1 = min(max(y1 - m.P, 0), H);   // the band's rows of the image proper
    int a[2], next_y[2], prev_y[2], after_y[2];
    unsigned long long left[2];   // seeds of the band not passed yet, a bit per row
    bool any[2];
    constexpr int FAR_BELOW = 0x3FFFFFFF, FAR_ABOVE = -0x3FFFFFFF;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        after_y[k] = FAR_BELOW;
        prev_y[k] = FAR_ABOVE;
        left[k] = 0;
        a[k] = 0;
        const int col = c + k - m.P;
        if (col >= 0 && col < W) {
            const long long b0 = m.bit0 + (long long)col * H + r0;
            const long long w0 = b0 >> 5;
            const int shift = (int)(b0 & 31), n = r1 - r0;
            if (r0 < H) {
                const uint32_t first = __ldg(&ranks.bits[w0]);
                a[k] = __ldg(&ranks.before[w0]) + __popc(first & ((1u << shift) - 1u));
                unsigned long long v = first >> shift;
                if (n + shift > 32) v |= (unsigned long long)__ldg(&ranks.bits[w0 + 1]) << (32 - shift);
                if (n + shift > 64) v |= (unsigned long long)__ldg(&ranks.bits[w0 + 2]) << (64 - shift);
                if (n < 64) v &= (1ull << n) - 1ull;
                left[k] = v << (m.P + r0 - y0 & 63);   // n rows from there on: none if the band lies above the image
            } else {   // below the image proper: the column's seeds are all above
                const long long end = m.bit0 + (long long)(col + 1) * H - 1, w = end >> 5;
                a[k] = __ldg(&ranks.before[w]) + __popc(__ldg(&ranks.bits[w]) & (0xFFFFFFFFu >> (31 - (int)(end & 31))));
            }
            const int x = m.ox + c + k, b = a[k] + __popcll(left[k]);
            if (b < m.s1) {
                const uint32_t p = __ldg(&pos[b]);
                if ((int)pos_x(p) == x) after_y[k] = (int)pos_y(p) - m.oy;
            }
            if (a[k] > m.s0) {
                const uint32_t p = __ldg(&pos[a[k] - 1]);
                if ((int)pos_x(p) == x) prev_y[k] = (int)pos_y(p) - m.oy;
            }
        }
        if (c + k < m.Wp)
            bands[m.band_off + band * m.Wp + c + k] =
                make_uint4((uint32_t)a[k], 0u, (uint32_t)left[k], (uint32_t)(left[k] >> 32));
        next_y[k] = left[k] ? y0 + __ffsll((long long)left[k]) - 1 : after_y[k];
        any[k] = next_y[k] != FAR_BELOW || prev_y[k] != FAR_ABOVE;
    }
    int16_t* dst = off + (size_t)(m.oy + y0) * pitch + m.ox + c;
    const bool paired = c + 1 < m.Wp && ((m.ox | pitch) & 1) == 0;   // c is even
    for (int y = y0; y < y1; ++y, dst += pitch) {
        int v[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (next_y[k] < y) {   // the seed below was passed: it becomes the one above
                prev_y[k] = next_y[k];
                left[k] &= left[k] - 1;
                next_y[k] = left[k] ? y0 + __ffsll((long long)left[k]) - 1 : after_y[k];
                ++a[k];
            }
            const int below = next_y[k] - y, above = y - prev_y[k];   // tie: the larger y, the higher rank
            bool down = below <= above;
            if (ranks.label && below == above && any[k])
                down = __ldg(&ranks.label[a[k]]) > __ldg(&ranks.label[a[k] - 1]);
            v[k] = any[k] ? (down ? below : -above) : NO_SEED;
        }
        if (paired) {
            *reinterpret_cast<short2*>(dst) = make_short2((short)v[0], (short)v[1]);
        } else {
            if (c < m.Wp) dst[0] = (int16_t)v[0];
            if (c + 1 < m.Wp) dst[1] = (int16_t)v[1];
        }
    }
}

// ---- row pass -----------------------------------------------------------
//
// With F_x = dy_x^2 + x^2 for each column x that has a candidate, the cell at
// column t takes the column minimising F_x - 2 t x (its squared distance minus
// t^2), ties to the larger x, the higher id.  All of it fits 32 bits: F_x <
// 2^31, 2 t x < 2^31 and F_x - 2 t x >= -t^2.
//  1. A column on or above the line between two others, one on each side, wins
//     no cell (only the vertices of the lower convex hull of the points
//     (x, F_x) do; on an edge the right end ties too).  Each warp thins out its
//     share of the columns: a parallel test of every column against its two
//     neighbours in the list, the survivors moved together, again and again
//     (the first pass tests three pairs).  4 096 columns go to 1 610, 962 and
//     665 in three passes at 200 000 uniform seeds (the hull has 559).
//     Whatever is left over costs time only.
//  2. A cell's winner never moves left as t grows, so the winners of the cells
//     1024 apart, then 256 apart, then 32 apart bound those in between: the
//     first two by a warp over the list range, the last by a lane each.
//  3. A warp takes 32 cells and tests the list between its two bounds, a
//     broadcast load and four instructions per column (unrolled by four, 2 %
//     of an image over the compiler's choice; by one or two was no better).
// The work is O(W) per row whatever the seed layout (the ranges of one step
// add up to the list and one column per cell looked at).  It is bound by
// instruction issue; a monotone chain per thread in step 1 (its pops diverge)
// took twice the instructions, merging such hulls pairwise left most lanes
// idle.
// Shared memory is 8 bytes per column, so that enough rows share an SM: the
// offsets, the columns' list, and room for W / 2 list entries with their F; a
// longer list (seed sets denser than one in ten cells, or a line of seeds across
// the image) keeps F and the columns in arrays of their own, and each cell looks
// its id up for itself (with F worked out again each time, 88 us instead of 71 at
// 2048 x 2048, one seed in three cells).  Rows of more than ROW_WIDE columns get 6 bytes per
// column, room for W / 4 entries; their longer lists hold columns only and work
// F out again each time.
constexpr int ROW_STEP = 32, ROW_MID = 256, ROW_TOP = 1024;
constexpr int ROW_THIN = 5;    // thinning passes at most
constexpr int ROW_WIDE = 27000;
constexpr int ROW_SHARE = 528;
// stands for a missing column's square: with any other it outweighs twice any
// real square, and two of them still fit
constexpr uint32_t NO_SQUARE = 0x7FFFFF00u;

inline int row_list_bytes(int W) { return W > ROW_WIDE ? 2 : 4; }   // per column, for the widest row of a launch
inline size_t row_pass_smem(int W)
{
    const size_t w = (size_t)(W + 7) / 4 * 4;
    return w * (4 + row_list_bytes(W)) + (size_t)(W / ROW_STEP + 3) * 4 + 16;
}
// Wide rows too few to fill the device take 32 warps each (one row of 32 767
// columns: 37 us against 72 with 8; 40 rows of 32 703: 43 against 86).
constexpr unsigned ROW_FEW = 148;
// Threads per row: warps of at most ROW_SHARE columns, up to 8 (twice that
// where there are rows enough to fill the device with fewer warps each: 678 us
// instead of 744 for a batch of 512 images; at 4 128 rows it is 136 against 129).
inline int row_pass_threads(int W, unsigned rows)
{
    const int share = rows >= 32768 ? 2 * ROW_SHARE : ROW_SHARE;
    if (rows <= ROW_FEW && W > 8 * ROW_SHARE) return 1024;
    return W <= share ? 32 : W <= 2 * share ? 64 : W <= 4 * share ? 128 : 256;
}

// Steps 2 and 3 of the row pass over a list of n columns; cost(k, t) is
// F - 2 t x of its entry k.  LABELS: ties between columns go to the higher
// label, whichever side it lies on; a cell's bounds are then the first minimum
// at the anchor before and the last one at the anchor after.
template <int T, bool LABELS, class Cost>
__device__ __forceinline__ void x_row_fill(const int2* list2, const uint16_t* listx, uint16_t* buf, uint16_t* hx,
                                           uint16_t* win, uint16_t* win_lo, const int16_t* off, int n, int W, int y,
                                           const XImg& m, const SeedBands& seeds, int32_t* __restrict__ out,
                                           Cost cost, bool packed)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = T / 32;
    auto sync = [] {
        if (T == 32) __syncwarp();
        else __syncthreads();
    };
    auto name = [&](int32_t rank) { return LABELS ? __ldg(&seeds.label[rank]) : rank; };
    auto by_warp = [&](int i, int lo, int hi) {
        const int t = i * ROW_STEP;
        int32_t best = 0x7FFFFFFF;
        int arg = lo, first = 0x7FFFFFFF;
#pragma unroll 4
        for (int k = lo + lane; k <= hi; k += 32) {
            const int32_t c = cost(k, t);
            if (LABELS && c < best) first = k;
            if (c <= best) {
                best = c;
                arg = k;
            }
        }
        const int32_t low = __reduce_min_sync(0xFFFFFFFFu, best);
        const int last = (int)__reduce_max_sync(0xFFFFFFFFu, best == low ? arg : -1);
        if (lane == 0) win[i] = (uint16_t)last;
        if (LABELS) {
            const int f = (int)__reduce_min_sync(0xFFFFFFFFu, best == low ? first : 0x7FFFFFFF);
            if (lane == 0) win_lo[i] = (uint16_t)f;
        }
    };
    const uint16_t* low = LABELS ? win_lo : win;

    // 2. winners of the cells ROW_TOP, ROW_MID and ROW_STEP apart
    const int steps = (W + ROW_STEP - 1) / ROW_STEP;
    constexpr int TOP = ROW_TOP / ROW_STEP, MID = ROW_MID / ROW_STEP;
    for (int i = warp * TOP; i < steps; i += NW * TOP) by_warp(i, 0, n - 1);
    if (tid == 0) win[steps] = (uint16_t)(n - 1);
    sync();
    for (int i = warp * MID; i < steps; i += NW * MID) {
        if (i % TOP == 0) continue;
        const int up = i / TOP * TOP;
        by_warp(i, low[up], win[min(up + TOP, steps)]);
    }
    sync();
    for (int i = tid; i < steps; i += T) {
        if (i % MID == 0) continue;
        const int up = i / MID * MID, hi = win[min(up + MID, steps)], t = i * ROW_STEP;
        int arg = low[up], first = arg;
        int32_t best = cost(arg, t);
#pragma unroll 4
        for (int k = arg + 1; k <= hi; ++k) {
            const int32_t c = cost(k, t);
            if (LABELS && c < best) first = k;
            if (c <= best) {
                best = c;
                arg = k;
            }
        }
        win[i] = (uint16_t)arg;
        if (LABELS) win_lo[i] = (uint16_t)first;
    }
    if (packed) {
        // labels of the listed columns' seeds: the offsets move aside first,
        // then buf and hx take the labels' halves (each list entry is one thread's)
        for (int k = tid; k < n; k += T) hx[k] = (uint16_t)off[list2[k].y / -2];
        sync();
        for (int k = tid; k < n; k += T) {
            const int32_t id = name(x_seed_at(seeds, m, m.ox + list2[k].y / -2, y + (int16_t)hx[k]));
            buf[k] = (uint16_t)(id & 0xFFFF);
            hx[k] = (uint16_t)(id >> 16);
        }
    }
    sync();
    auto label_of = [&](int k) -> int32_t {
        if (packed) return (int32_t)buf[k] | (int32_t)hx[k] << 16;
        const int x = listx[k];
        return name(x_seed_at(seeds, m, m.ox + x, y + off[x]));
    };

    // 3. every cell, from the list between its interval's bounds
    for (int i = warp; i < steps; i += NW) {
        const int t = i * ROW_STEP + lane;
        const int hi = win[i + 1];
        int arg = low[i];
        int32_t best = cost(arg, t);
#pragma unroll 4
        for (int k = arg + 1; k <= hi; ++k) {
            const int32_t c = cost(k, t);
            if (LABELS ? c < best || (c == best && label_of(k) > label_of(arg)) : c <= best) {
                best = c;
                arg = k;
            }
        }
        if (t < W) out[t] = label_of(arg);
    }
}

// row: the row's offsets; y: its row on the plane; out: its labels;
// list_bytes: row_list_bytes of the launch.
template <int T, bool LABELS>
__device__ __forceinline__ void x_row(const int16_t* __restrict__ row, int y, const XImg& m, const SeedBands& seeds,
                                      int32_t* __restrict__ out, int list_bytes)
{
    extern __shared__ __align__(16) unsigned char row_smem[];
    __shared__ int s_sum[T / 32 + 1];
    const int W = m.Wp;
    const int w = (W + 7) / 4 * 4;
    const int cap = w * list_bytes / 8;                            // (F, -2 x) entries that fit
    int2* list2 = reinterpret_cast<int2*>(row_smem);
    uint16_t* listx = reinterpret_cast<uint16_t*>(row_smem);       // the longer list
    uint16_t* buf = reinterpret_cast<uint16_t*>(row_smem + (size_t)w * list_bytes);   // offsets, then id low halves
    uint16_t* hx = buf + w;                                        // columns kept, then id high halves
    uint16_t* win = hx + w;                                        // winner at each 32nd cell
    uint16_t* win_lo = win + (W / ROW_STEP + 3);                   // LABELS: the first of the tied ones
    constexpr int TIE = LABELS ? 1 : 0;   // columns that could still tie are kept
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = T / 32;
    auto sync = [] {
        if (T == 32) __syncwarp();
        else __syncthreads();
    };

    // the row's offsets, by aligned words (an odd start brings one cell of its
    // left neighbour along)
    const int skew = (int)((reinterpret_cast<uintptr_t>(row) >> 1) & 1);
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(row - skew);
        uint32_t* dst = reinterpret_cast<uint32_t*>(buf);
        for (int i = tid; i < (W + skew + 1) / 2; i += T) dst[i] = __ldg(&src[i]);
    }
    const int16_t* off = reinterpret_cast<const int16_t*>(buf) + skew;
    sync();
    auto value = [&](int x) {
        const int d = off[x];
        return d * d + x * x;
    };

    // 1. each warp thins its share of the columns [s0, s1) into hx[s0, s0 + kept)
    const int share = ((W + NW - 1) / NW + 31) / 32 * 32;
    const int s0 = min(W, warp * share), s1 = min(W, s0 + share);
    const unsigned below = (1u << lane) - 1u;
    int kept = 0;
    // the first test, four columns a lane, against the columns 1, 2 and 4 to
    // either side (at equal distances k it is d_l^2 + d_r^2 + 2 k^2 <= 2 d_x^2)
    for (int base = s0; base < s1; base += 128) {
        const int x = base + 4 * lane;
        uint32_t q[12];   // squares of columns x - 4 .. x + 7; beyond the warp's 128: not there
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int d = x + c < W ? off[x + c] : NO_SEED;
            q[4 + c] = d == NO_SEED ? NO_SQUARE : (uint32_t)(d * d);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t l = __shfl_up_sync(0xFFFFFFFFu, q[4 + c], 1);
            const uint32_t r = __shfl_down_sync(0xFFFFFFFFu, q[4 + c], 1);
            q[c] = lane > 0 ? l : NO_SQUARE;
            q[8 + c] = lane < 31 ? r : NO_SQUARE;
        }
        int at = s0 + kept, total = 0;
        bool keep[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t d = q[4 + c], dd = 2u * d;
            keep[c] = x + c < s1 && d != NO_SQUARE && q[3 + c] + q[5 + c] + 2u + TIE > dd &&
                      q[2 + c] + q[6 + c] + 8u + TIE > dd && q[c] + q[8 + c] + 32u + TIE > dd;
            const unsigned k = __ballot_sync(0xFFFFFFFFu, keep[c]);
            at += __popc(k & below);
            total += __popc(k);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (keep[c]) hx[at++] = (uint16_t)(x + c);
        kept += total;
    }
    __syncwarp();
    for (int pass = 1; pass < ROW_THIN && kept > 2; ++pass) {
        // in place: a group's writes stay at or before its own reads, and
        // reach a later group's left neighbour only where nothing was dropped
        int now = 0;
        for (int base = 0; base < kept; base += 32) {
            const int i = base + lane;
            bool keep = i < kept;
            int x = 0;
            if (keep) {
                x = hx[s0 + i];
                if (i > 0 && i + 1 < kept) {
                    const int xl = hx[s0 + i - 1], xr = hx[s0 + i + 1];
                    const int32_t f = value(x), fl = value(xl), fr = value(xr);
                    keep = (long long)(x - xl) * (fr - f) + TIE > (long long)(f - fl) * (xr - x);
                }
            }
            const unsigned k = __ballot_sync(0xFFFFFFFFu, keep);
            __syncwarp();
            if (keep) hx[s0 + now + __popc(k & below)] = (uint16_t)x;
            now += __popc(k);
            __syncwarp();
        }
        const bool settled = kept - now < kept / 8;
        kept = now;
        if (settled) break;
    }
    // one list of all of them
    int at = 0, n = kept;
    if (T > 32) {
        if (lane == 0) s_sum[warp] = kept;
        __syncthreads();
        n = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            const int v = s_sum[k];
            at += k < warp ? v : 0;
            n += v;
        }
    }
    const bool packed = n <= cap;
    for (int j = lane; j < kept; j += 32) {
        const int x = hx[s0 + j];
        if (packed) list2[at + j] = make_int2(value(x), -2 * x);
        else listx[at + j] = (uint16_t)x;
    }
    sync();
    if (n == 0) {
        for (int t = tid; t < W; t += T) out[t] = UNDEF;
        return;
    }
    if (packed) {
        x_row_fill<T, LABELS>(list2, listx, buf, hx, win, win_lo, off, n, W, y, m, seeds, out,
                              [&](int k, int t) {
            const int2 c = list2[k];
            return c.x + t * c.y;
        }, true);
    } else if (list_bytes == 4) {   // room for any list: the columns move on to hx, F takes their place
        int32_t* listf = reinterpret_cast<int32_t*>(row_smem);
        for (int k = tid; k < n; k += T) hx[k] = listx[k];
        sync();
        for (int k = tid; k < n; k += T) listf[k] = value(hx[k]);
        sync();
        x_row_fill<T, LABELS>(list2, hx, buf, hx, win, win_lo, off, n, W, y, m, seeds, out,
                              [&](int k, int t) { return listf[k] - 2 * t * (int)hx[k]; }, false);
    } else {
        x_row_fill<T, LABELS>(list2, listx, buf, hx, win, win_lo, off, n, W, y, m, seeds, out,
                              [&](int k, int t) {
            const int x = listx[k];
            return value(x) - 2 * t * x;
        }, false);
    }
}

}  // namespace idl
