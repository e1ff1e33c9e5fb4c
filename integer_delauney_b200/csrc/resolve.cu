// Stage (a), reference semantics from scratch, without iterating: the Jacobi
// fixed point read off the exact diagram.
//
// The reference's iteration (src/cuda/voronoi.cu:32-53,100-113) starts from
// the seed cells and ends where no neighbour's owner beats a cell's own.  At
// 4096 x 4096 with 200 000 uniform seeds it takes 51 passes and its result
// differs from the exact diagram (exact.cu) in 2 933 of 17 M cells.  Which
// cells, and what they hold, follows from a few local rules, so the passes
// need not be run.
//
// Write e(q) for a cell's exact owner (nearest seed, ties to the higher id),
// |q - s| for the L1 distance, and "k displays at q at time t" for "the
// iteration's label of q after t passes is k".  Keys only improve, a cell
// takes the best of its own and its neighbours' labels, and a label moves one
// cell per pass, so k cannot be at q before t = |q - k|.
//
//  (1) Settled cells.  If a monotone 4-path leads from q to its owner's cell
//      through cells of the same exact owner, the owner arrives at every cell
//      of the path at its L1 distance and stays: nothing beats it there.  So
//      q displays e(q) from A(q) = |q - e(q)| on, for good.  Every cell with a
//      settled neighbour of its own owner one step nearer the owner is
//      settled; a cell with no same-owner neighbour on the way is a root, and
//      the roots with the cells that reach their owner only through roots are
//      the suspects (k_roots, k_suspects): 3 034 cells at the size above.
//      They are the tips of thin Voronoi regions, cut off on the grid.
//  (2) A suspect p ends with the best label its neighbours ever display: at
//      least f, the best owner of its settled neighbours (by p's distances).
//      Only a seed that beats f at p can change that; those candidates are
//      the seeds in the disc through f around p, found column by column from
//      the column pass's plane.  Best candidate first:
//      (no)  k never reaches p if a search from p, through cells where k could
//            still be displayed, meets no settled cell of k.  k can be
//            displayed at r only from |r - k| on, only before A(r), and only
//            until a better owner of a settled neighbour m of r arrives, at
//            A(m) + 1.
//      (yes) k reaches p if, along a digital line from p to k, every cell q up
//            to the first settled cell of k is beyond every better seed m of
//            q at the time k gets there: |q - m| > |q - k|.  Then k displays
//            at each q at time |q - k| exactly.  (The segment from p to its
//            exact owner lies inside the owner's region, so the cells of the
//            line leave that region by less than a cell.)
//      97 % of the suspects end at "no" on the first step, nearly all others
//      at "yes" within 3 cells (40 with clustered seeds).  Where both fail,
//      each is tried once more with the other's help: a better seed that
//      certainly arrives at r in time closes r to k, and one that never
//      arrives at q does not count there.
//  (3) What that leaves (suspects with no settled neighbour: none at the size
//      above, a few among seeds on a circle) is stepped: the iteration itself
//      on a WIN x WIN window around p in shared memory, restricted to the
//      cells whose label can still matter to p at a time when it is not known
//      (k_resolve_window).  If such cells reach the
//      window's edge, or a list overflows, resolve_fail is raised and the
//      caller runs the pass-by-pass propagation instead; the kernels that
//      follow, and what is left of the one at work, then end at once.
//
// The kernels' results are checked against the iteration on uniform, clustered,
// lattice, line and circle seed sets by the GPU tests.
//
// Cost at 4096 x 4096, 200 000 uniform seeds: one read of the label plane for
// the roots (37 us, bound by the latency of its loads), the suspects 8 us, their
// decisions 28 to 42 us (a chain of dependent loads per suspect, 3 034 of them;
// the worst one's decides), the rest 6 us.  With the exact diagram's 160 us that
// is 0.25 ms of propagation; the 51 passes took 1.18 ms.  With 200 000 clustered
// seeds 0.28 ms, the 1 100 passes 7.8 ms.
// Where the passes have to run after all, the attempt comes on top of them: 2 to
// 14 % of a call (seeds on circles, a spiral, a parabola of 2 048 x 2 048), most
// of it the decisions of the cells that could be decided.
#include "context.cuh"
#include "exact_pass.cuh"
#include "stencil.cuh"

#include <atomic>

namespace idl {
namespace {

struct View {
    const int32_t* lab;      // exact labels
    const int16_t* off;      // column pass: row offset to the nearest seed of the cell's column
    SeedBands seeds;         // and its table
    const uint32_t* pos;     // seed positions by label
    const uint32_t* sorted;  // and by (x, y) rank
    const uint32_t* sus;     // suspect bits, rows of `words` words
    const XImg* images;      // batch: image table, else null
    const int32_t* seed_img; // batch: image of each seed
    int pitch, Wd, Hd, words;
    XImg whole;              // not a batch: the one image
};

__device__ __forceinline__ int sgn(int v) { return (v > 0) - (v < 0); }

__device__ __forceinline__ int32_t label_at(const View& V, int x, int y)
{
    return (x >= 0 && y >= 0 && x < V.Wd && y < V.Hd) ? __ldg(&V.lab[(size_t)y * V.pitch + x]) : OUTSIDE;
}

// (x, y) inside the canvas; V.sus is complete when this is used
__device__ __forceinline__ bool suspect_at(const View& V, int x, int y)
{
    return (__ldg(&V.sus[(size_t)y * V.words + (x >> 5)]) >> (x & 31)) & 1u;
}

__device__ __forceinline__ int l1_to(const View& V, int x, int y, int32_t s)
{
    const uint32_t p = __ldg(&V.pos[s]);
    return abs(x - pos_x(p)) + abs(y - pos_y(p));
}

__device__ __forceinline__ int32_t d2_to(const View& V, int x, int y, int32_t s)
{
    return dist2(x, y, __ldg(&V.pos[s]));
}

__device__ __forceinline__ bool beats(int32_t da, int32_t a, int32_t db, int32_t b)
{
    return da < db || (da == db && a > b);
}

__device__ __forceinline__ int isqrt(int32_t v)   // floor, v >= 0
{
    int r = (int)sqrtf((float)v);
    while ((long long)r * r > v) --r;
    while ((long long)(r + 1) * (r + 1) <= v) ++r;
    return r;
}

// ---- (1) roots and suspects -------------------------------------------

// A warp takes 128 columns (four per lane) by ROOT_ROWS rows, loaded at once
// with the rows above and below; cells that their neighbours' owners rule out
// are skipped without a seed-table load.
constexpr int ROOT_ROWS = 8;

__global__ void __launch_bounds__(128)
k_roots(const int32_t* __restrict__ lab, int pitch, int Wd, int Hd, const uint32_t* __restrict__ pos,
        uint32_t* __restrict__ sus, int words, int32_t* __restrict__ list, int cap, Scalars* __restrict__ sc)
{
    __shared__ uint16_t queue[4][ROOT_ROWS * 128];
    const int lane = threadIdx.x & 31;
    const int x0 = (blockIdx.x * 32 + lane) * 4;
    const int y0 = (blockIdx.y * 4 + (threadIdx.x >> 5)) * ROOT_ROWS;
    if (y0 >= Hd) return;
    int4 v[ROOT_ROWS + 2];
    int32_t edge[ROOT_ROWS];   // lane 0: the cell left of the warp's columns, lane 31: right of them
#pragma unroll
    for (int j = 0; j < ROOT_ROWS + 2; ++j) {
        const int y = y0 + j - 1;
        const bool in = y >= 0 && y < Hd && x0 < Wd;   // rows are padded to a multiple of 32 columns
        const int32_t* p = lab + (size_t)y * pitch + x0;
        v[j] = in ? __ldg(reinterpret_cast<const int4*>(p)) : make_int4(OUTSIDE, OUTSIDE, OUTSIDE, OUTSIDE);
        if (j >= 1 && j <= ROOT_ROWS)
            edge[j - 1] = in && lane == 0 && x0 > 0 ? __ldg(p - 1)
                          : in && lane == 31 && x0 + 4 < Wd ? __ldg(p + 4) : OUTSIDE;
    }
    // A cell in its owner's row or column is linked: the next cell on the way is
    // on the segment between them, inside the owner's region.  So a root has a
    // differing neighbour both across and up or down; of those (a quarter of
    // the cells at 200 000 seeds in 4096 x 4096) the owner's direction decides.
    unsigned maybe = 0;   // bit 4 row + column of the lane's cells
#pragma unroll
    for (int j = 1; j <= ROOT_ROWS; ++j) {
        const int4 up = v[j - 1], cur = v[j], dn = v[j + 1];
        int32_t lf = __shfl_up_sync(FULL, cur.w, 1), rt = __shfl_down_sync(FULL, cur.x, 1);
        if (lane == 0) lf = edge[j - 1];
        if (lane == 31) rt = edge[j - 1];
        const int32_t row[6] = {lf, cur.x, cur.y, cur.z, cur.w, rt};
        const int32_t above[4] = {up.x, up.y, up.z, up.w}, below[4] = {dn.x, dn.y, dn.z, dn.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int32_t s = row[c + 1];
            const bool across = row[c] != s || row[c + 2] != s, along = above[c] != s || below[c] != s;
            if (s >= 0 && across && along) maybe |= 1u << (4 * (j - 1) + c);
        }
    }
    const int valid = min(max(Wd - x0, 0), 4);
    if (valid < 4) maybe &= 0x11111111u * ((1u << valid) - 1u);
    // worked off 32 at a time from a queue, so that the seed table is read with full warps
    uint16_t* q = queue[threadIdx.x >> 5];
    const int mine = __popc(maybe);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += u;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    for (int at = incl - mine; maybe; ++at) {
        const int i = __ffs(maybe) - 1;
        maybe &= maybe - 1;
        q[at] = (uint16_t)((i >> 2) * 128 + lane * 4 + (i & 3));
    }
    __syncwarp();
    for (int i = lane; i < total; i += 32) {
        const int x = blockIdx.x * 128 + q[i] % 128, y = y0 + q[i] / 128;
        const int32_t* p = lab + (size_t)y * pitch + x;
        const int32_t s = __ldg(p);
        const uint32_t o = __ldg(&pos[s]);
        const int dx = pos_x(o) - x, dy = pos_y(o) - y;
        // the neighbours one step nearer the owner lie on the canvas, like the owner
        const bool linked = dx == 0 || dy == 0 || __ldg(p + sgn(dx)) == s || __ldg(p + (long long)sgn(dy) * pitch) == s;
        if (!linked) {
            atomicOr(&sus[(size_t)y * words + (x >> 5)], 1u << (x & 31));
            const int k = atomicAdd(&sc->n_roots, 1);
            if (k < cap) list[k] = (int32_t)pack_pos(x, y);
        }
    }
}

// For the pass count: the largest A of a settled cell into sc->arrive_max.  On
// the finished labels, of which the settled cells' are their exact owners still.
__global__ void __launch_bounds__(256)
k_arrivals(const int32_t* __restrict__ lab, int pitch, int Wd, int Hd, const uint32_t* __restrict__ pos,
           const uint32_t* __restrict__ sus, int words, Scalars* __restrict__ sc)
{
    int far = 0;
    for (int y = blockIdx.x; y < Hd; y += gridDim.x)
        for (int x = threadIdx.x; x < Wd; x += 256) {
            const int32_t l = __ldg(&lab[(size_t)y * pitch + x]);
            const uint32_t w = __ldg(&sus[(size_t)y * words + (x >> 5)]);
            if (l < 0 || ((w >> (x & 31)) & 1u)) continue;
            const uint32_t p = __ldg(&pos[l]);
            far = max(far, abs((int)pos_x(p) - x) + abs((int)pos_y(p) - y));
        }
    far = __reduce_max_sync(FULL, far);
    if ((threadIdx.x & 31) == 0) atomicMax(&sc->arrive_max, far);
}

// The cells that reach their owner only through roots.  A cell is suspect
// once all its same-owner neighbours nearer the owner are; whichever thread
// marks the last of those sees the others' bits (mark, fence, look), so each
// thread follows what it marked itself.
__global__ void __launch_bounds__(128)
k_suspects(View V, uint32_t* sus, int32_t* list, int cap, Scalars* sc)
{
    const int n = sc->n_roots;
    if (n > cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) sc->resolve_fail = 1;
        return;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        constexpr int DEPTH = 24;
        uint32_t stack[DEPTH];
        int top = 0;
        stack[top++] = (uint32_t)list[i];
        while (top > 0) {
            const uint32_t c = stack[--top];
            const int cx = pos_x(c), cy = pos_y(c);
            const int32_t s = label_at(V, cx, cy);
            const uint32_t p = __ldg(&V.pos[s]);
            for (int j = 0; j < 4; ++j) {
                const int x = cx + (j == 0) - (j == 1), y = cy + (j == 2) - (j == 3);
                if (label_at(V, x, y) != s) continue;
                const int dx = sgn(pos_x(p) - x), dy = sgn(pos_y(p) - y);
                if (dx == 0 && dy == 0) continue;
                // only a cell one step further out than c can hang on c
                if (!((x + dx == cx && y == cy) || (x == cx && y + dy == cy))) continue;
                auto marked = [&](int mx, int my) {
                    return (atomicOr(&sus[(size_t)my * V.words + (mx >> 5)], 0u) >> (mx & 31)) & 1u;
                };
                if (dx && label_at(V, x + dx, y) == s && !marked(x + dx, y)) continue;
                if (dy && label_at(V, x, y + dy) == s && !marked(x, y + dy)) continue;
                const uint32_t bit = 1u << (x & 31);
                if (atomicOr(&sus[(size_t)y * V.words + (x >> 5)], bit) & bit) continue;
                __threadfence();
                const int k = n + atomicAdd(&sc->n_more, 1);
                if (k < cap && top < DEPTH) {
                    list[k] = (int32_t)pack_pos(x, y);
                    stack[top++] = pack_pos(x, y);
                } else {
                    sc->resolve_fail = 1;
                }
            }
        }
    }
}

// ---- (2) deciding a suspect -------------------------------------------

constexpr int RES_WARPS = 4;
constexpr int MAX_CAND = 16;    // candidates of one suspect, rivals at one cell (2 at most at the sizes above)
// Cells of a "no" search: 32, 64 and 128 take the same time and leave the same
// cells open on every set measured.  The first, short one is not sharp either: 8,
// 16 and 32 cells 72, 76 and 83 us at 200 000 clustered seeds, 855, 882 and 937
// between lines of seeds.
constexpr int MAX_SEARCH = 64;
constexpr int SHORT_SEARCH = 16;
constexpr int MAX_FRONT = 4;    // line cells per step (2 are reached)
// Disc columns (in warp strides) a suspect may look at: 1 600 are reached with
// clustered seeds, 10 536 between lines of seeds across 4096 x 4096 (all decided;
// with 2^12 they would run the passes, 2^16 costs the same); beyond it the suspect
// stays undecided, so that no seed set makes a warp run long: 4 ms.
constexpr int BUDGET = 1 << 14;
constexpr int LONG_SPENT = 256;

// resolve_fail as it is now, the same for all lanes of the warp.
__device__ __forceinline__ bool raised(const Scalars* sc, int lane)
{
    const int v = lane == 0 ? __ldcg(&sc->resolve_fail) : 0;
    return __shfl_sync(FULL, v, 0) != 0;
}

struct WarpScratch {
    int32_t cand[MAX_CAND], rival[2][MAX_CAND];
    uint32_t seen[2][MAX_SEARCH];
    int n, n_rival, budget;
    const Scalars* sc;
};

// Offers every seed m of the image that beats (d, s) at (x, y) to f(m); a lane
// takes every 32nd column.  The column pass's plane gives each column's
// nearest seed at row y; its neighbours in id order are the column's other
// seeds.  f returns false to stop the lane.
template <class F>
__device__ __forceinline__ void for_better(const View& V, int x, int y, int32_t d, int32_t s, const XImg& b, int lane,
                                           F&& f)
{
    const int R = isqrt(d);
    const int lo = max(b.ox, x - R), hi = min(b.ox + b.Wp - 1, x + R);
    const int16_t* row = V.off + (size_t)y * V.pitch;
    for (int x0 = lo + lane; x0 <= hi; x0 += 128) {
        int o[4];   // four columns' loads in flight: a disc of the empty parts of a clustered set has a thousand
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = x0 + 32 * j <= hi ? __ldg(&row[x0 + 32 * j]) : NO_SEED;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int xx = x0 + 32 * j;
            if (o[j] == NO_SEED || (long long)o[j] * o[j] + (long long)(xx - x) * (xx - x) > d) continue;
            const int32_t c = x_seed_at(V.seeds, b, xx, y + o[j]);
            for (int step = 1; step >= -1; step -= 2) {
                for (int32_t r = step > 0 ? c : c - 1; r >= b.s0 && r < b.s1; r += step) {
                    const uint32_t p = __ldg(&V.sorted[r]);
                    if ((int)pos_x(p) != xx) break;   // past the column's run
                    const int32_t dm = dist2(x, y, p);
                    if (dm > d) break;
                    const int32_t m = V.seeds.label ? __ldg(&V.seeds.label[r]) : r;
                    if (m != s && beats(dm, m, d, s) && !f(m, p)) return;
                }
            }
        }
    }
}

// Can k still be displayed at the cell (x, y) = r?  (rule "no")
__device__ __forceinline__ bool may_display(const View& V, int x, int y, int32_t l, bool sus, int32_t k)
{
    const int t = l1_to(V, x, y, k);
    if (!sus && l1_to(V, x, y, l) <= t) return false;   // settled with its own owner by then
    const int32_t dk = d2_to(V, x, y, k);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int mx = x + (j == 0) - (j == 1), my = y + (j == 2) - (j == 3);
        const int32_t m = label_at(V, mx, my);
        if (m < 0 || m == k || suspect_at(V, mx, my)) continue;
        if (beats(d2_to(V, x, y, m), m, dk, k) && l1_to(V, mx, my, m) < t) return false;
    }
    return true;
}

__device__ __forceinline__ XImg image_of(const View& V, int32_t seed)
{
    return V.images ? V.images[V.seed_img[seed]] : V.whole;
}

// S.rival[LEVEL]: the seeds that beat k at (x, y) and can be there by the time
// k can (|q - m| <= |q - k|); their number, above MAX_CAND if they do not fit or the
// budget is spent.
template <int LEVEL>
__device__ __forceinline__ int rivals(const View& V, WarpScratch& S, int x, int y, int32_t k, const XImg& b, int lane)
{
    const int t = l1_to(V, x, y, k);
    const int32_t d = d2_to(V, x, y, k);
    __syncwarp();
    if (lane == 0) {
        S.n_rival = 0;
        S.budget -= 1 + (isqrt(d) >> 4);
        // a long decision (1 % of them with clustered seeds) ends with the others
        if (S.budget < BUDGET - LONG_SPENT && __ldcg(&S.sc->resolve_fail)) S.budget = -1;
    }
    __syncwarp();
    if (S.budget < 0) return MAX_CAND + 1;
    for_better(V, x, y, d, k, b, lane, [&](int32_t m, uint32_t mp) {
        if (abs(x - (int)pos_x(mp)) + abs(y - (int)pos_y(mp)) > t) return true;
        const int at = atomicAdd(&S.n_rival, 1);
        if (at < MAX_CAND) S.rival[LEVEL][at] = m;
        return at < MAX_CAND;
    });
    __syncwarp();
    return S.n_rival;
}

template <int LEVEL>
__device__ bool never(const View& V, WarpScratch& S, int px, int py, int32_t k, const XImg& b, int lane,
                      int cap = MAX_SEARCH);

// Rule "yes": k certainly arrives at (px, py), at its L1 distance.  LEVEL 1: a
// rival that never arrives at a cell does not count there.  Warp-wide.
template <int LEVEL>
__device__ bool arrives(const View& V, WarpScratch& S, int px, int py, int32_t k, const XImg& b, int lane)
{
    const uint32_t kp = __ldg(&V.pos[k]);
    const int gx = sgn((int)pos_x(kp) - px), gy = sgn((int)pos_y(kp) - py);
    const int DX = abs((int)pos_x(kp) - px), DY = abs((int)pos_y(kp) - py);
    int front[MAX_FRONT] = {}, nf = 1;   // steps in x of the cells reached s steps from p
    for (int s = 1; s <= DX + DY && nf > 0; ++s) {
        int next[MAX_FRONT] = {}, nn = 0;
        for (int a = 0; a < nf; ++a) {
            for (int d = 0; d < 2; ++d) {
                const int u = front[a] + d, v = s - u;
                if (u > DX || v > DY) continue;
                if (llabs((long long)u * DY - (long long)v * DX) >= DX + DY) continue;
                bool dup = false;
                for (int w = 0; w < nn; ++w) dup = dup || next[w] == u;
                if (dup) continue;
                const int x = px + gx * u, y = py + gy * v;
                const int32_t l = label_at(V, x, y);
                const bool su = suspect_at(V, x, y);
                if (!su && l == k) return true;
                if (!su && l1_to(V, x, y, l) <= DX + DY - s) continue;
                const int nr = rivals<LEVEL>(V, S, x, y, k, b, lane);
                bool pass = nr == 0 || (LEVEL > 0 && nr <= MAX_CAND);
                if (LEVEL > 0)
                    for (int q = 0; pass && q < nr; ++q) pass = never<0>(V, S, x, y, S.rival[LEVEL][q], b, lane);
                if (pass && nn < MAX_FRONT) next[nn++] = u;
            }
        }
        nf = nn;
        for (int w = 0; w < MAX_FRONT; ++w) front[w] = next[w];
    }
    return false;
}

// Rule "no": k certainly never arrives at (px, py).  LEVEL 1: a cell where a
// rival of k certainly arrives no later than k can is closed to k.  Warp-wide.
// The search takes eight cells at a time, four lanes each; it gives up beyond
// `cap` cells.
template <int LEVEL>
__device__ bool never(const View& V, WarpScratch& S, int px, int py, int32_t k, const XImg& b, int lane, int cap)
{
    uint32_t* seen = S.seen[LEVEL];
    int ns = 1, head = 0;
    __syncwarp();
    if (lane == 0) seen[0] = pack_pos(px, py);
    __syncwarp();
    const int dir = lane & 3;
    while (head < ns) {
        const int at = head + (lane >> 2);
        head = min(head + 8, ns);
        bool src = false, add = false;
        int x = 0, y = 0;
        if (at < head) {
            const uint32_t q = seen[at];
            x = (int)pos_x(q) + (dir == 0) - (dir == 1);
            y = (int)pos_y(q) + (dir == 2) - (dir == 3);
            const int32_t l = label_at(V, x, y);
            if (l >= 0) {
                const bool su = suspect_at(V, x, y);
                src = !su && l == k;
                if (!src) {
                    bool old = false;
                    for (int w = 0; w < ns; ++w) old = old || seen[w] == pack_pos(x, y);
                    add = !old && may_display(V, x, y, l, su, k);
                }
            }
        }
        if (__any_sync(FULL, src)) return false;
        // a cell two of them lead to is taken once
        const unsigned same = __match_any_sync(FULL, add ? pack_pos(x, y) : 0xFFFFFFFFu);
        unsigned ab = __ballot_sync(FULL, add && lane == __ffs(same) - 1);
        if (LEVEL > 0) {
            for (unsigned m = ab; m; m &= m - 1) {
                const int j = __ffs(m) - 1;
                const int rx = __shfl_sync(FULL, x, j), ry = __shfl_sync(FULL, y, j);
                const int nr = rivals<LEVEL>(V, S, rx, ry, k, b, lane);
                if (nr > MAX_CAND) return false;
                bool closed = false;
                for (int c = 0; !closed && c < nr; ++c) closed = arrives<0>(V, S, rx, ry, S.rival[LEVEL][c], b, lane);
                if (closed) ab &= ~(1u << j);
            }
        }
        if (ns + __popc(ab) > cap) return false;
        if ((ab >> lane) & 1u) seen[ns + __popc(ab & ((1u << lane) - 1u))] = pack_pos(x, y);
        ns += __popc(ab);
        __syncwarp();
    }
    return true;
}

// Appends suspect i to the open ones.
__device__ __forceinline__ void leave_open(int i, int32_t* open, int open_cap, Scalars* sc)
{
    const int at = atomicAdd(&sc->n_open, 1);
    if (at < open_cap) open[at] = i;
    else sc->resolve_fail = 1;
}

// One warp per suspect.  res[i] takes the final label, or -1 with i appended
// to `open` (at most open_cap) for the window kernel.  The time of p's last change is at least
// its label's L1 distance (sc->arrive_max) and at most sc->late_max.
__global__ void __launch_bounds__(RES_WARPS * 32, 4)
k_resolve(View V, const int32_t* __restrict__ list, int32_t* __restrict__ res, int32_t* __restrict__ open,
          int open_cap, Scalars* __restrict__ sc)
{
    __shared__ WarpScratch scratch[RES_WARPS];
    WarpScratch& S = scratch[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int n = sc->n_roots + sc->n_more;
    if (__any_sync(FULL, sc->resolve_fail)) return;   // read with the counts
    if (lane == 0) S.sc = sc;
    // More suspects than warps: those without a settled neighbour go first, since
    // too many of them end the run.
    if (n > (int)gridDim.x * RES_WARPS) {
        for (int i = blockIdx.x * RES_WARPS * 32 + threadIdx.x; i < n; i += gridDim.x * RES_WARPS * 32) {
            const uint32_t pk = (uint32_t)list[i];
            bool settled = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int x = (int)pos_x(pk) + (j == 0) - (j == 1), y = (int)pos_y(pk) + (j == 2) - (j == 3);
                settled = settled || (label_at(V, x, y) >= 0 && !suspect_at(V, x, y));
            }
            if (!settled) leave_open(i, open, open_cap, sc);
        }
        __syncwarp();
    }
    for (int i = blockIdx.x * RES_WARPS + (threadIdx.x >> 5); i < n; i += gridDim.x * RES_WARPS) {
        if (n > (int)gridDim.x * RES_WARPS && raised(sc, lane)) return;
        const uint32_t pk = (uint32_t)list[i];
        const int px = pos_x(pk), py = pos_y(pk);
        const XImg b = image_of(V, label_at(V, px, py));
        // f: the best owner of the settled neighbours
        int32_t f = -1, fd = FAR;
        int f_at = 0;   // when the settled neighbour holding f displays it, plus one
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = px + (j == 0) - (j == 1), y = py + (j == 2) - (j == 3);
            const int32_t m = label_at(V, x, y);
            if (m < 0 || suspect_at(V, x, y)) continue;
            const int32_t d = d2_to(V, px, py, m);
            const int at = l1_to(V, x, y, m) + 1;
            if (m == f) f_at = min(f_at, at);
            else if (f < 0 || beats(d, m, fd, f)) {
                f = m;
                fd = d;
                f_at = at;
            }
        }
        bool decided = f >= 0;
        int32_t out = f;
        int t_hi = f_at;
        if (decided) {
            if (lane == 0) {
                S.n = 0;
                S.budget = BUDGET;
            }
            __syncwarp();
            for_better(V, px, py, fd, f, b, lane, [&](int32_t m, uint32_t) {
                const int at = atomicAdd(&S.n, 1);
                if (at < MAX_CAND) S.cand[at] = m;
                return at < MAX_CAND;
            });
            __syncwarp();
            const int nc = S.n;
            decided = nc <= MAX_CAND;
            int32_t last = 0x7FFFFFFF, last_d = -1;   // the candidate just ruled out
            for (int c = 0; decided && c < nc; ++c) {
                // the best candidate after `last`
                int32_t k = -1, kd = FAR;
                for (int q = 0; q < nc; ++q) {
                    const int32_t m = S.cand[q];
                    const int32_t d = d2_to(V, px, py, m);
                    if (last_d >= 0 && !beats(last_d, last, d, m)) continue;
                    if (k < 0 || beats(d, m, kd, k)) {
                        k = m;
                        kd = d;
                    }
                }
                last = k;
                last_d = kd;
                // a short search, then the line, which is quick where it succeeds
                if (never<0>(V, S, px, py, k, b, lane, SHORT_SEARCH)) continue;
                const bool yes = arrives<0>(V, S, px, py, k, b, lane);
                if (!yes && (never<0>(V, S, px, py, k, b, lane) || never<1>(V, S, px, py, k, b, lane))) continue;
                if (yes || arrives<1>(V, S, px, py, k, b, lane)) {
                    out = k;
                    t_hi = l1_to(V, px, py, k);
                } else {
                    decided = false;
                }
                break;
            }
        }
        if (lane == 0) {
            res[i] = decided ? out : -1;
            if (decided) {
                const int t_lo = l1_to(V, px, py, out);
                atomicMax(&sc->arrive_max, t_lo);
                atomicMax(&sc->late_max, t_hi);
            } else if (out >= 0 || n <= (int)gridDim.x * RES_WARPS) {   // without a settled neighbour: open already
                leave_open(i, open, open_cap, sc);
            }
        }
        __syncwarp();
    }
}

// ---- (3) the undecided, stepped in a window ---------------------------

// need[q]: the latest time at which q's label is not known beforehand and
// still matters to p (-1: none).  p's own label matters throughout; if q's
// label matters at time t, its neighbours' matter at t - 1.  A settled cell
// is known from A on, and no cell holds any label before ceil(its distance
// to its nearest seed).  Cells with need >= 0 are stepped; the others show
// their owner from A on and nothing before, which is right whenever asked.
constexpr int WIN = 96;
constexpr int WIN_THREADS = 512;
static_assert(4 * WIN <= WIN_THREADS, "a thread per cell of the window's sides");
constexpr int WIN_N = WIN * WIN;
constexpr size_t WIN_SMEM = (size_t)WIN_N * (4 * 4 + 2 * 2);
constexpr int32_t FOREVER = 1 << 28;

__global__ void __launch_bounds__(WIN_THREADS)
k_resolve_window(View V, const int32_t* __restrict__ list, const int32_t* __restrict__ open,
                 int32_t* __restrict__ res, Scalars* __restrict__ sc)
{
    extern __shared__ __align__(16) int32_t win[];
    int32_t* own = win;                 // exact labels, OUTSIDE / walls negative
    int32_t* st0 = own + WIN_N;         // state, two buffers
    int32_t* st1 = st0 + WIN_N;
    volatile int32_t* need = st1 + WIN_N;
    uint16_t* arr = reinterpret_cast<uint16_t*>(st1 + 2 * WIN_N);   // A, 0xFFFF for a suspect
    uint16_t* first = arr + WIN_N;      // no label before this time
    __shared__ int s_t0, s_t1, s_bad, s_stop;
    const int n = sc->n_open;   // beyond the list only with resolve_fail raised
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        if (threadIdx.x == 0) s_stop = __ldcg(&sc->resolve_fail);
        __syncthreads();
        if (s_stop) return;
        const int i = open[it];
        const uint32_t pk = (uint32_t)list[i];
        const int ox = (int)pos_x(pk) - WIN / 2, oy = (int)pos_y(pk) - WIN / 2;
        const int ctr = (WIN / 2) * WIN + WIN / 2;
        if (threadIdx.x == 0) {
            s_t0 = FOREVER;
            s_t1 = 0;
            s_bad = 0;
        }
        for (int c = threadIdx.x; c < WIN_N; c += WIN_THREADS) {
            const int x = ox + c % WIN, y = oy + c / WIN;
            const int32_t l = label_at(V, x, y);
            own[c] = l;
            st0[c] = st1[c] = UNDEF;
            need[c] = c == ctr ? FOREVER : -1;
            uint16_t a = 0xFFFF, fr = 0xFFFF;
            if (l >= 0) {
                if (!suspect_at(V, x, y)) a = (uint16_t)min(l1_to(V, x, y, l), 0xFFFE);
                const int32_t d = d2_to(V, x, y, l);
                const int r = isqrt(d);
                fr = (uint16_t)(r + ((long long)r * r < d));
            }
            arr[c] = a;
            first[c] = fr;
        }
        __syncthreads();
        // need, to its fixed point (values only grow, each bounded by a neighbour's - 1)
        for (int sweep = 0; sweep < 4 * WIN_N; ++sweep) {
            bool ch = false;
            for (int c = threadIdx.x; c < WIN_N; c += WIN_THREADS) {
                if (own[c] < 0) continue;
                const int cx = c % WIN, cy = c / WIN;
                int m = -1;
                if (cx > 0) m = max(m, need[c - 1] - 1);
                if (cx < WIN - 1) m = max(m, need[c + 1] - 1);
                if (cy > 0) m = max(m, need[c - WIN] - 1);
                if (cy < WIN - 1) m = max(m, need[c + WIN] - 1);
                if (arr[c] != 0xFFFF) m = min(m, (int)arr[c] - 1);
                if (m >= (int)first[c] && m > need[c]) {
                    need[c] = m;
                    ch = true;
                }
            }
            if (!__syncthreads_or(ch)) break;
            if (sweep % 8 == 7) {   // a stepped cell at the window's edge: found again below, no need to go on
                bool edge = threadIdx.x == 0 && __ldcg(&sc->resolve_fail);
                if (threadIdx.x < 4 * WIN) {
                    const int side = threadIdx.x / WIN, at = threadIdx.x % WIN;
                    const int cx = side == 0 ? 0 : side == 1 ? WIN - 1 : at, cy = side == 2 ? 0 : side == 3 ? WIN - 1 : at;
                    edge = edge || (need[cy * WIN + cx] >= 0 &&
                                    label_at(V, ox + cx + (side == 1) - (side == 0),
                                             oy + cy + (side == 3) - (side == 2)) >= 0);
                }
                if (__syncthreads_or(edge)) break;
            }
        }
        // the stepped cells must lie inside the window; their time span
        for (int c = threadIdx.x; c < WIN_N; c += WIN_THREADS) {
            if (need[c] < 0) continue;
            const int cx = c % WIN, cy = c / WIN, x = ox + cx, y = oy + cy;
            if ((cx == 0 && label_at(V, x - 1, y) >= 0) || (cx == WIN - 1 && label_at(V, x + 1, y) >= 0) ||
                (cy == 0 && label_at(V, x, y - 1) >= 0) || (cy == WIN - 1 && label_at(V, x, y + 1) >= 0))
                s_bad = 1;
            atomicMin(&s_t0, (int)first[c]);
            for (int j = 0; j < 5; ++j) {   // the last time a cell it reads settles
                const int nx = cx + (j == 0) - (j == 1), ny = cy + (j == 2) - (j == 3);
                if (nx < 0 || ny < 0 || nx >= WIN || ny >= WIN) continue;
                const int a = arr[ny * WIN + nx];
                if (a != 0xFFFF) atomicMax(&s_t1, a);
            }
        }
        __syncthreads();
        if (s_bad) {
            if (threadIdx.x == 0) sc->resolve_fail = 1;
            __syncthreads();
            continue;
        }
        // step from the first time any label can show until all settled cells
        // have settled and a step changes nothing
        int32_t* cur = st0;
        int32_t* nxt = st1;
        int last = 0;
        bool done = false;
        const int t_end = s_t1 + 2 + WIN_N;
        for (int t = s_t0; t <= t_end; ++t) {   // cur: time t - 1
            bool ch = false;
            for (int c = threadIdx.x; c < WIN_N; c += WIN_THREADS) {
                if (need[c] < 0) continue;
                const int cx = c % WIN, cy = c / WIN, x = ox + cx, y = oy + cy;
                auto shown = [&](int q) {   // label of q at time t - 1
                    if (own[q] < 0) return UNDEF;
                    if (arr[q] != 0xFFFF && t - 1 >= (int)arr[q]) return own[q];
                    return need[q] >= 0 ? cur[q] : UNDEF;
                };
                const int32_t was = shown(c);
                int32_t k = was, d = k >= 0 ? d2_to(V, x, y, k) : FAR;
                if (cx > 0) relax(k, d, shown(c - 1), x, y, V.pos);
                if (cx < WIN - 1) relax(k, d, shown(c + 1), x, y, V.pos);
                if (cy > 0) relax(k, d, shown(c - WIN), x, y, V.pos);
                if (cy < WIN - 1) relax(k, d, shown(c + WIN), x, y, V.pos);
                nxt[c] = k;
                if (k != was) {
                    ch = true;
                    if (c == ctr) last = t;
                }
            }
            ch = __syncthreads_or(ch);
            int32_t* tb = cur;
            cur = nxt;
            nxt = tb;
            if (!ch && t > s_t1 + 1) {
                done = true;
                break;
            }
        }
        if (last > 0) atomicMax(&sc->arrive_max, last);
        if (threadIdx.x == 0) {
            if (done) res[i] = cur[ctr];
            else sc->resolve_fail = 1;
        }
        __syncthreads();
    }
}

__global__ void k_resolve_apply(int32_t* __restrict__ lab, int pitch, const int32_t* __restrict__ list,
                                const int32_t* __restrict__ res, const Scalars* __restrict__ sc)
{
    if (sc->resolve_fail) return;
    const int n = sc->n_roots + sc->n_more;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t p = (uint32_t)list[i];
        if (res[i] >= 0) lab[(size_t)pos_y(p) * pitch + pos_x(p)] = res[i];
    }
}

}  // namespace

bool resolved(Context& C)
{
    const Scalars& s = *C.host_sc;
    int64_t* count = C.selftest.count;
    ++count[s.resolve_fail ? IDL_COUNT_PASSES : IDL_COUNT_DIRECT];
    if (!s.resolve_fail) count[IDL_COUNT_WINDOWS] += s.n_open;
    return !s.resolve_fail;
}

size_t resolve_reserve(Context& C, const Canvas& cv)
{
    const size_t bits = (size_t)ceil_div(cv.Wd, 32) * cv.Hd * 4;
    C.sus_bits.ensure(bits);
    return bits;
}

void resolve_exact(Context& C, const Canvas& cv, const uint32_t* pos, int64_t n, const XImg* images,
                   const int32_t* seed_img, const uint32_t* sorted, const int32_t* label)
{
    if (C.prof.enabled) C.prof.prop_bytes += (double)cv.Wd * cv.Hd * 4.0;   // labels in, for the roots
    const int words = ceil_div(cv.Wd, 32);
    const size_t bits = resolve_reserve(C, cv);
    // suspects: 0.02 % of the cells at the usual densities (at most 0.4 % in
    // the densest sets measured); beyond the lists the iteration takes over
    const int cap = (int)C.selftest.bound(IDL_LIMIT_SUSPECTS,
                                          std::min<int64_t>((int64_t)cv.Wd * cv.Hd / 64 + 4096, 1 << 22));
    C.sus_list.ensure((size_t)cap * 3 * 4);
    int32_t* list = C.sus_list.as<int32_t>();
    int32_t* res = list + cap;
    int32_t* open = res + cap;
    uint32_t* sus = C.sus_bits.as<uint32_t>();
    if (!C.precleared) {
        IDL_CUDA(cudaMemsetAsync(sus, 0, bits, C.stream));
        IDL_CUDA(cudaMemsetAsync(&C.sc()->n_roots, 0, RESOLVE_SCALARS * sizeof(int32_t), C.stream));
    }
    const View V{C.lab[0].as<int32_t>(), C.lab[1].as<int16_t>(), SeedBands{C.exact_bands.as<uint4>(), label}, pos,
                 sorted ? sorted : pos, sus, images,
                 seed_img, cv.pitch, cv.Wd, cv.Hd, words, whole_canvas(cv, n, 0)};
    const dim3 g((unsigned)ceil_div(cv.Wd, 128), (unsigned)ceil_div(cv.Hd, 4 * ROOT_ROWS));
    k_roots<<<g, 128, 0, C.stream>>>(V.lab, cv.pitch, cv.Wd, cv.Hd, pos, sus, words, list, cap, C.sc());
    IDL_LAUNCH();
    const int gs = std::max(1, std::min(ceil_div(cap, 128), C.num_sms));
    k_suspects<<<gs, 128, 0, C.stream>>>(V, sus, list, cap, C.sc());
    IDL_LAUNCH();
    // a window takes up to a millisecond, the passes a few at most: a batch gets
    // four windows per SM; an image with more than a few (seeds on a wide circle,
    // a hundred and more) does not fit them either
    const int open_cap = (int)C.selftest.bound(IDL_LIMIT_OPEN, std::min(cap, images ? C.num_sms * 4 : 64));
    k_resolve<<<std::min(ceil_div(cap, RES_WARPS), C.num_sms * 8), RES_WARPS * 32, 0, C.stream>>>(V, list, res, open,
                                                                                              open_cap, C.sc());
    IDL_LAUNCH();
    static std::atomic<uint64_t> opted{0};   // the shared-memory opt-in is per device
    const uint64_t bit = 1ull << (C.device & 63);
    if (!(opted.load(std::memory_order_acquire) & bit)) {
        IDL_CUDA(cudaFuncSetAttribute((const void*)k_resolve_window, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)WIN_SMEM));
        opted.fetch_or(bit, std::memory_order_acq_rel);
    }
    k_resolve_window<<<std::min(open_cap, C.num_sms), WIN_THREADS, WIN_SMEM, C.stream>>>(V, list, open, res, C.sc());
    IDL_LAUNCH();
    k_resolve_apply<<<gs, 256, 0, C.stream>>>(C.lab[0].as<int32_t>(), cv.pitch, list, res, C.sc());
    IDL_LAUNCH();
}

void resolve_arrivals(Context& C, const Canvas& cv, const uint32_t* pos)
{
    k_arrivals<<<std::min(cv.Hd, C.num_sms * 8), 256, 0, C.stream>>>(C.lab[0].as<int32_t>(), cv.pitch, cv.Wd, cv.Hd, pos,
                                                                    C.sus_bits.as<uint32_t>(), ceil_div(cv.Wd, 32),
                                                                    C.sc());
    IDL_LAUNCH();
}

}  // namespace idl
