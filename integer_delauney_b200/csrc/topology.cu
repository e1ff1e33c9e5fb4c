// Stage (b): Delaunay triangles from 2x2 label blocks, deduplicated and
// numbered canonically, entirely on the device.
//
// The rule (src/cuda/triangle_detect.cuh:75-166): a block whose four labels
// hold three distinct seeds witnesses one triangle, emitted in first-seen
// order; four distinct seeds are a degree-4 Voronoi vertex, cut along the
// shorter diagonal of the quad ordered cyclically around its centroid, ties
// going to the diagonal that avoids the lowest seed id; any UNDEF label skips
// the block.  The reference orders the quad with double-precision atan2; here
// the order is exact integer arithmetic that sorts the same way atan2's
// values do (see angle_less), so no transcendental is needed.
//
// Dedup and numbering.  The reference appends 32-byte records through one
// global atomic counter, sorts them with thrust::sort, uniques them and copies
// them to the host (triangulation.cu:229-271); which duplicate survives is up
// to the unstable sort.  Here each emitted triangle goes straight into an
// open-addressing hash table keyed by its sorted vertex triple packed in 63
// bits (21 bits per id, as delaunay.cuh:372-374 packs it); the value kept per
// key is an atomicMin over (row-major block index, vertex order), so the
// witness is the first block in scan order, deterministically.  Canonical ids
// (rank of the sorted triple, what thrust::sort(RawLess) yields,
// triangulation.cu:254) come from grouping keys by their smallest vertex: a
// count per seed, an exclusive scan, and a rank within each (tiny) group.
#include "context.cuh"

namespace idl {
namespace {

constexpr unsigned long long EMPTY_KEY = ~0ull;
constexpr int MAX_PROBES = 1 << 14;

__device__ __forceinline__ unsigned long long mix64(unsigned long long k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

// atan2(v.y, v.x) < atan2(u'.y, u'.x) decided exactly for integer vectors.
// atan2 maps to (-pi, pi]: y < 0 gives (-pi, 0), (x >= 0, y == 0) gives 0
// (the zero vector included, atan2(+0, +0) = +0), y > 0 gives (0, pi) and
// (x < 0, y == 0) gives pi.  Within the two open half planes the order is
// the sign of the cross product.
__device__ __forceinline__ int angle_class(int x, int y)
{
    if (y < 0) return 0;
    if (y == 0) return x >= 0 ? 1 : 3;
    return 2;
}

__device__ __forceinline__ bool angle_less(int ax, int ay, int bx, int by)
{
    const int ca = angle_class(ax, ay), cb = angle_class(bx, by);
    if (ca != cb) return ca < cb;
    if (ca == 1 || ca == 3) return false;
    return (long long)ax * by - (long long)ay * bx > 0;
}

struct Emit {
    int32_t o0[3], o1[3];
    int n;
};

template <class V>
__device__ __forceinline__ V pick(int i, V a, V b, V c, V d)
{
    return i == 0 ? a : i == 1 ? b : i == 2 ? c : d;
}

// The block rule of triangle_detect.cuh:75-166 on labels (a, b, c, d) =
// (top-left, top-right, bottom-left, bottom-right).  Written without indexed
// arrays, so that everything stays in registers.
__device__ __forceinline__ void block_rule(int32_t a, int32_t b, int32_t c, int32_t d,
                                           const uint32_t* __restrict__ pos, Emit& e)
{
    e.n = 0;
    if ((a | b | c | d) < 0) return;
    const int same = (a == b) + (a == c) + (a == d) + (b == c) + (b == d) + (c == d);
    if (same > 1) return;
    if (same == 1) {   // three labels, in first-seen order
        const bool bb = b == a, cc = c == a || c == b;
        e.o0[0] = a;
        e.o0[1] = bb ? c : b;
        e.o0[2] = bb || cc ? d : c;
        e.n = 1;
        return;
    }
    const uint32_t p0 = __ldg(&pos[a]), p1 = __ldg(&pos[b]), p2 = __ldg(&pos[c]), p3 = __ldg(&pos[d]);
    const int x0 = pos_x(p0), x1 = pos_x(p1), x2 = pos_x(p2), x3 = pos_x(p3);
    const int y0 = pos_y(p0), y1 = pos_y(p1), y2 = pos_y(p2), y3 = pos_y(p3);
    const int sx = x0 + x1 + x2 + x3, sy = y0 + y1 + y2 + y3;
    // 4 * (p - centroid), exact in integers
    const int vx0 = 4 * x0 - sx, vx1 = 4 * x1 - sx, vx2 = 4 * x2 - sx, vx3 = 4 * x3 - sx;
    const int vy0 = 4 * y0 - sy, vy1 = 4 * y1 - sy, vy2 = 4 * y2 - sy, vy3 = 4 * y3 - sy;
    // places in the stable order by angle: a later one goes first only if strictly less
    const bool l10 = angle_less(vx1, vy1, vx0, vy0), l20 = angle_less(vx2, vy2, vx0, vy0),
               l30 = angle_less(vx3, vy3, vx0, vy0), l21 = angle_less(vx2, vy2, vx1, vy1),
               l31 = angle_less(vx3, vy3, vx1, vy1), l32 = angle_less(vx3, vy3, vx2, vy2);
    const int r0 = l10 + l20 + l30, r1 = !l10 + l21 + l31, r2 = !l20 + !l21 + l32, r3 = !l30 + !l31 + !l32;
    auto at_rank = [&](int r) { return r0 == r ? 0 : r1 == r ? 1 : r2 == r ? 2 : r3 == r ? 3 : 3; };
    const int o0 = at_rank(0), o1 = at_rank(1), o2 = at_rank(2), o3 = at_rank(3);
    auto len2 = [&](int i, int j) {
        const int dx = pick(i, x0, x1, x2, x3) - pick(j, x0, x1, x2, x3);
        const int dy = pick(i, y0, y1, y2, y3) - pick(j, y0, y1, y2, y3);
        return (uint32_t)(dx * dx) + (uint32_t)(dy * dy);
    };
    const uint32_t l0 = len2(o0, o2), l1 = len2(o1, o3);
    bool first = l0 < l1;   // the diagonal o0 - o2
    if (l0 == l1) {
        const int lowest = a < b && a < c && a < d ? 0 : b < c && b < d ? 1 : c < d ? 2 : 3;
        first = !(lowest == o0 || lowest == o2);
    }
    const int pa = first ? o0 : o1, pb = first ? o2 : o3;
    const int u = first ? o1 : o0, v = first ? o3 : o2;
    const int ra = min(u, v), rb = max(u, v);
    e.o0[0] = e.o1[0] = pick(pa, a, b, c, d);
    e.o0[1] = e.o1[1] = pick(pb, a, b, c, d);
    e.o0[2] = pick(ra, a, b, c, d);
    e.o1[2] = pick(rb, a, b, c, d);
    e.n = 2;
}

// Sorted key plus a 4-bit code of the order the block saw the vertices in.
// With a rank map the key and the recorded ids are ranks (the numbering the
// outputs use) while the rule itself ran on the raw labels.
__device__ __forceinline__ void make_key(const int32_t in[3], const int32_t* __restrict__ rank, unsigned long long& key,
                                         unsigned& code)
{
    const int32_t o[3] = {rank ? __ldg(&rank[in[0]]) : in[0], rank ? __ldg(&rank[in[1]]) : in[1],
                          rank ? __ldg(&rank[in[2]]) : in[2]};
    int32_t a = o[0], b = o[1], c = o[2], t;
    if (a > b) { t = a; a = b; b = t; }
    if (b > c) { t = b; b = c; c = t; }
    if (a > b) { t = a; a = b; b = t; }
    key = ((unsigned long long)a << 42) | ((unsigned long long)b << 21) | (unsigned long long)c;
    const unsigned i0 = o[0] == a ? 0u : (o[0] == b ? 1u : 2u);
    const unsigned i1 = o[1] == a ? 0u : (o[1] == b ? 1u : 2u);
    code = i0 * 3u + i1;
}

// The table interleaves each slot's key and value (table[2s], table[2s + 1]),
// so an insert touches one 16-byte pair in one memory sector.
__device__ __forceinline__ void hash_insert(unsigned long long key, unsigned long long val,
                                            unsigned long long* __restrict__ table, unsigned long long mask,
                                            Scalars* __restrict__ sc)
{
    unsigned long long slot = mix64(key) & mask;
    for (int probe = 0; probe < MAX_PROBES; ++probe) {
        const unsigned long long prev = atomicCAS(&table[2 * slot], EMPTY_KEY, key);
        if (prev == EMPTY_KEY || prev == key) {
            atomicMin(&table[2 * slot + 1], val);
            return;
        }
        slot = (slot + 1) & mask;
    }
    atomicOr(&sc->overflow, 1);
}

__device__ __forceinline__ void detect_block(const int32_t* __restrict__ lab, int pitch, int Wd,
                                             const uint32_t* __restrict__ pos, const int32_t* __restrict__ rank,
                                             int x, int y, unsigned long long* __restrict__ table,
                                             unsigned long long mask, Scalars* __restrict__ sc)
{
    const int32_t* p = lab + (size_t)y * pitch + x;
    Emit e;
    block_rule(p[0], p[1], p[pitch], p[pitch + 1], pos, e);
    const unsigned long long blk = (unsigned long long)y * Wd + x;
    unsigned long long key;
    unsigned code;
    if (e.n > 0) {
        make_key(e.o0, rank, key, code);
        hash_insert(key, (blk << 4) | code, table, mask, sc);
    }
    if (e.n > 1) {
        make_key(e.o1, rank, key, code);
        hash_insert(key, (blk << 4) | code, table, mask, sc);
    }
}

// A warp covers a strip of DET_COLS x DET_ROWS blocks (2 x 2 cells each, by
// their top-left cell): four columns per lane, the label rows streaming
// through registers, so that the plane is read once and a block costs a few
// comparisons.  The blocks with three or four labels (one in forty at 200 000
// seeds in 4096 x 4096) go into a queue in shared memory first and are worked
// off 32 at a time: run in place, the rule and the table's round trips occupy
// a whole warp for the one or two lanes that have a vertex.  A strip with more
// than DET_OWN of them (a dense blob) leaves the others to k_detect_rest, which
// spreads them over the device.
// 46 us at that size (126 with a thread per block), bound by the latency of the
// loads and of the table's round trips: 25 % of HBM bandwidth, 49 % issue.
// Canvases too small to fill the device with such strips use shorter ones.
constexpr int DET_COLS = 128, DET_ROWS = 16, DET_ROWS_SMALL = 4, DET_WARPS = 4, DET_OWN = 96;
static_assert(DET_ROWS * 4 == 64, "a lane's blocks are the bits of one 64-bit mask");

template <int ROWS>
__global__ void __launch_bounds__(DET_WARPS * 32)
k_detect(const int32_t* __restrict__ lab, int pitch, int Wd, int Hd, const uint32_t* __restrict__ pos,
         const int32_t* __restrict__ rank, unsigned long long* __restrict__ table, unsigned long long mask,
         Scalars* __restrict__ sc, uint32_t* __restrict__ rest, int rest_cap)
{
    __shared__ uint16_t queue[DET_WARPS][DET_COLS * ROWS];
    uint16_t* q = queue[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int xs = blockIdx.x * DET_COLS, ys = (blockIdx.y * DET_WARPS + (threadIdx.x >> 5)) * ROWS;
    if (ys >= Hd - 1) return;
    const int x0 = xs + lane * 4;
    // one row's five labels: the lane's four columns and the next (rows are
    // padded to a multiple of 32 columns; blocks beyond Wd - 1 are masked out;
    // a row past the canvas has none).  Four rows are loaded at a time.
    auto load = [&](int y, int4& v, int32_t& edge) {
        const int32_t* p = lab + (size_t)y * pitch + x0;
        const bool in = y < Hd && x0 < Wd;
        v = in ? __ldg(reinterpret_cast<const int4*>(p)) : make_int4(-1, -1, -1, -1);
        edge = in && lane == 31 && x0 + 4 < Wd ? __ldg(p + 4) : -1;
    };
    int4 up;
    int32_t up_edge;
    load(ys, up, up_edge);
    int32_t up_next = __shfl_down_sync(0xffffffffu, up.x, 1);
    if (lane == 31) up_next = up_edge;
    unsigned long long hit = 0;
#pragma unroll
    for (int r0 = 0; r0 < ROWS; r0 += 4) {
        int4 v[4];
        int32_t edge[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) load(ys + r0 + j + 1, v[j], edge[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int4 dn = v[j];
            int32_t dn_next = __shfl_down_sync(0xffffffffu, dn.x, 1);
            if (lane == 31) dn_next = edge[j];
            const int32_t u[5] = {up.x, up.y, up.z, up.w, up_next}, d[5] = {dn.x, dn.y, dn.z, dn.w, dn_next};
            unsigned here = 0;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int32_t A = u[c], B = u[c + 1], C = d[c], D = d[c + 1];
                // three or four different labels: at most one of the six pairs is equal
                const int same = (A == B) + (C == D) + (A == C) + (B == D) + (A == D) + (B == C);
                if (same <= 1 && (A | B | C | D) >= 0) here |= 1u << c;
            }
            hit |= (unsigned long long)here << (4 * (r0 + j));
            up = dn;
            up_next = dn_next;
        }
    }
    // columns whose block has no right cell
    const int valid = min(max(Wd - 1 - x0, 0), 4);
    if (valid < 4) hit &= 0x1111111111111111ull * ((1u << valid) - 1u);
    const int mine = __popcll(hit);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int at = incl - mine; hit; ++at) {
        const int b = __ffsll((long long)hit) - 1;
        hit &= hit - 1;
        q[at] = (uint16_t)((b >> 2) * DET_COLS + lane * 4 + (b & 3));
    }
    __syncwarp();
    for (int i = lane; i < min(total, DET_OWN); i += 32)
        detect_block(lab, pitch, Wd, pos, rank, xs + q[i] % DET_COLS, ys + q[i] / DET_COLS, table, mask, sc);
    if (total <= DET_OWN) return;
    int at = lane == 0 ? atomicAdd(&sc->n_blocks, total - DET_OWN) : 0;
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int i = DET_OWN + lane; i < total; i += 32) {
        const int x = xs + q[i] % DET_COLS, y = ys + q[i] / DET_COLS, k = at + i - DET_OWN;
        if (k < rest_cap) rest[k] = pack_pos(x, y);
        else detect_block(lab, pitch, Wd, pos, rank, x, y, table, mask, sc);
    }
}

__global__ void __launch_bounds__(128)
k_detect_rest(const int32_t* __restrict__ lab, int pitch, int Wd, const uint32_t* __restrict__ pos,
              const int32_t* __restrict__ rank, unsigned long long* __restrict__ table, unsigned long long mask,
              Scalars* __restrict__ sc, const uint32_t* __restrict__ rest, int rest_cap)
{
    const int n = min(sc->n_blocks, rest_cap);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        detect_block(lab, pitch, Wd, pos, rank, pos_x(rest[i]), pos_y(rest[i]), table, mask, sc);
}

// Compaction of the occupied slots with one atomic per block on the row
// counter (one per warp, 65 k of them on a 2 M-slot table, serialised on that
// one address): a block counts the occupied slots of its contiguous span,
// reserves that many rows, and writes them in slot order, the second read of
// the span coming from L2.  Row order is free: k_rank numbers the triangles
// canonically.
constexpr int ENUM_THREADS = 256;

__global__ void __launch_bounds__(ENUM_THREADS)
k_enumerate(const unsigned long long* __restrict__ table, long long cap, unsigned long long* __restrict__ ukeys,
            unsigned long long* __restrict__ uvals, int32_t* __restrict__ cnt, Scalars* __restrict__ sc)
{
    constexpr int NW = ENUM_THREADS / 32;
    __shared__ int warp_cnt[NW];
    __shared__ unsigned long long s_base;
    const long long span = ((cap + gridDim.x - 1) / gridDim.x + ENUM_THREADS - 1) / ENUM_THREADS * ENUM_THREADS;
    const long long b0 = (long long)blockIdx.x * span, b1 = min(cap, b0 + span);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned mine = 0;
    for (long long s = b0 + threadIdx.x; s < b1; s += ENUM_THREADS) mine += table[2 * s] != EMPTY_KEY;
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) warp_cnt[warp] = (int)mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int w = 0; w < NW; ++w) total += (unsigned)warp_cnt[w];
        s_base = total ? atomicAdd(reinterpret_cast<unsigned long long*>(&sc->n_triangles), total) : 0ull;
    }
    __syncthreads();
    unsigned long long base = s_base;
    for (long long s0 = b0; s0 < b1; s0 += ENUM_THREADS) {
        const long long s = s0 + threadIdx.x;
        const unsigned long long k = s < b1 ? table[2 * s] : EMPTY_KEY;
        const bool occ = k != EMPTY_KEY;
        const unsigned ballot = __ballot_sync(0xffffffffu, occ);
        if (lane == 0) warp_cnt[warp] = __popc(ballot);
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const int c = warp_cnt[w];
            before += w < warp ? c : 0;
            all += c;
        }
        if (occ) {
            const unsigned long long u = base + before + __popc(ballot & ((1u << lane) - 1u));
            ukeys[u] = k;
            uvals[u] = table[2 * s + 1];
            atomicAdd(&cnt[(int)(k >> 42)], 1);
        }
        base += all;
        __syncthreads();   // warp_cnt is rewritten next iteration
    }
}

__global__ void k_group(const unsigned long long* __restrict__ ukeys, const Scalars* __restrict__ sc,
                        const int32_t* __restrict__ off, int32_t* __restrict__ fill, int32_t* __restrict__ grp)
{
    const long long nu = sc->n_triangles;
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < nu;
         u += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(ukeys[u] >> 42);
        const int slot = atomicAdd(&fill[a], 1);
        grp[off[a] + slot] = (int32_t)u;
    }
}

__global__ void k_rank(const unsigned long long* __restrict__ ukeys, const unsigned long long* __restrict__ uvals,
                       const Scalars* __restrict__ sc, const int32_t* __restrict__ off,
                       const int32_t* __restrict__ grp, int Wd, int shift, int32_t* __restrict__ tris)
{
    const long long nu = sc->n_triangles;
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < nu;
         u += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = ukeys[u];
        const int a = (int)(k >> 42);
        const int lo = off[a], hi = off[a + 1];
        int r = 0;
        for (int j = lo; j < hi; ++j) r += ukeys[grp[j]] < k;
        const long long tid = lo + r;
        const int32_t id[3] = {(int32_t)(k >> 42), (int32_t)((k >> 21) & 0x1FFFFF), (int32_t)(k & 0x1FFFFF)};
        const unsigned long long v = uvals[u];
        const unsigned code = (unsigned)(v & 15u);
        const unsigned long long blk = v >> 4;
        const unsigned i0 = code / 3u, i1 = code % 3u, i2 = 3u - i0 - i1;
        int32_t* o = tris + tid * 5;
        o[0] = (int32_t)(blk % (unsigned long long)Wd) - shift;
        o[1] = (int32_t)(blk / (unsigned long long)Wd) - shift;
        o[2] = id[i0];
        o[3] = id[i1];
        o[4] = id[i2];
    }
}

}  // namespace

int64_t detect_capacity(const Context& C, int64_t n)
{
    // Unique triangles of a planar triangulation number under 2n; the table
    // starts at four times that (a table half that size probes longer: 17 us
    // more at 200 000 seeds), and on the rare probe
    // overflow it grows and the detection is redone.  The occupied slots are
    // counted while they are compacted (one atomic per block), not while they
    // are inserted, where a single counter would serialise every new key.
    const int64_t cap = std::max<int64_t>(next_pow2(8 * n + 1024), C.hash_cap);
    return next_pow2(C.selftest.bound(IDL_LIMIT_TABLE, cap));
}

void detect_reserve(Context& C, int64_t n, int64_t cap)
{
    C.cnt.ensure((size_t)(n + 1) * 2 * 4);   // counts, then fill positions: cleared together
    C.off.ensure((size_t)(n + 2) * 4);
    C.hkeys.ensure((size_t)cap * 16);
    C.ukeys.ensure((size_t)cap * 8);
    C.uvals.ensure((size_t)cap * 8);
    // grouping and ranking follow with no read-back between: their
    // buffers hold as many triangles as the table has slots, and their
    // count comes from the device
    C.grp.ensure((size_t)cap * 4);
    C.tris.ensure((size_t)cap * 5 * 4);
}

void detect_launch(Context& C, const Canvas& cv, const int32_t* labels, const uint32_t* pos, int64_t n, int shift,
                   int64_t cap, cudaEvent_t mid, const int32_t* rank)
{
    detect_reserve(C, n, cap);
    int32_t* cnt = C.cnt.as<int32_t>();
    int32_t* fill = cnt + n + 1;
    unsigned long long* table = C.hkeys.as<unsigned long long>();
    unsigned long long* ukeys = C.ukeys.as<unsigned long long>();
    unsigned long long* uvals = C.uvals.as<unsigned long long>();
    // the blocks left to k_detect_rest wait in the grouping buffer, free until then
    uint32_t* rest = C.grp.as<uint32_t>();
    static_assert(offsetof(Scalars, overflow) == 12 && offsetof(Scalars, n_blocks) == 8, "cleared together");
    if (!C.precleared) {
        ClearList l;
        l.add(table, (size_t)cap * 16, 0xFFFFFFFFu);
        l.add(C.scalars.ptr, 16, 0);   // n_triangles, n_blocks, overflow
        l.add(cnt, (size_t)(n + 1) * 2 * 4, 0);
        clear_buffers(C, l);
    }

    const int strips = ceil_div(std::max(cv.Wd - 1, 1), DET_COLS);
    const bool small = strips * ceil_div(cv.Hd, DET_ROWS) < C.num_sms * 16;
    const dim3 grd(strips, ceil_div(std::max(cv.Hd - 1, 1), (small ? DET_ROWS_SMALL : DET_ROWS) * DET_WARPS));
    auto* detect = small ? k_detect<DET_ROWS_SMALL> : k_detect<DET_ROWS>;
    detect<<<grd, DET_WARPS * 32, 0, C.stream>>>(labels, cv.pitch, cv.Wd, cv.Hd, pos, rank, table,
                                                 (unsigned long long)(cap - 1), C.sc(), rest, (int)cap);
    IDL_LAUNCH();
    k_detect_rest<<<C.num_sms * 4, 128, 0, C.stream>>>(labels, cv.pitch, cv.Wd, pos, rank, table,
                                                      (unsigned long long)(cap - 1), C.sc(), rest, (int)cap);
    IDL_LAUNCH();
    if (mid) IDL_CUDA(cudaEventRecord(mid, C.stream));
    C.mark(PM_DETECT);
    const int g1 = (int)std::min<int64_t>(ceil_div(cap, 256), C.num_sms * 16);
    k_enumerate<<<g1, ENUM_THREADS, 0, C.stream>>>(table, cap, ukeys, uvals, cnt, C.sc());
    IDL_LAUNCH();
    exclusive_scan(C, cnt, C.off.as<int32_t>(), n);
    const int g2 = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(2 * n + 2, 256), C.num_sms * 16));
    k_group<<<g2, 256, 0, C.stream>>>(ukeys, C.sc(), C.off.as<int32_t>(), fill, C.grp.as<int32_t>());
    IDL_LAUNCH();
    k_rank<<<g2, 256, 0, C.stream>>>(ukeys, uvals, C.sc(), C.off.as<int32_t>(), C.grp.as<int32_t>(), cv.Wd, shift,
                                     C.tris.as<int32_t>());
    IDL_LAUNCH();
}

bool detect_done(Context& C, int64_t cap)
{
    if (C.host_sc->overflow) return false;
    // keep the next run's table at most half full
    C.hash_cap = C.host_sc->n_triangles > cap / 2 ? cap * 4 : cap;
    return true;
}

void detect_triangles(Context& C, const Canvas& cv, const int32_t* labels, const uint32_t* pos, int64_t n,
                      int shift, cudaEvent_t mid, const int32_t* rank)
{
    int64_t cap = detect_capacity(C, n);
    for (int attempt = 0;; ++attempt) {
        detect_launch(C, cv, labels, pos, n, shift, cap, mid, rank);
        // one read-back: overflow (then all of it again, with a larger table) and the count
        C.fetch_scalars();
        if (detect_done(C, cap)) break;
        if (attempt >= 6) throw Error(IDL_ERR_INTERNAL, "triangle hash table overflow");
        cap *= 4;
    }
}

}  // namespace idl
