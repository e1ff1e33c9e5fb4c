// Batched triangulation: many independent images of uneven size and seed
// count through one pass of the pipeline.  Each image's result equals
// idl_triangulate on that image alone, bit for bit.
//
// The images' padded detection canvases are shelf-packed into one atlas with
// a one-cell wall between neighbours.  Wall cells hold a label below UNDEF,
// which the propagation never updates and never takes as a candidate, and
// which makes the block rule skip every 2x2 block touching it, so no image
// sees another.  Seeds get global ids image after image, each image's in its
// own (x asc, y asc) order, so within an image the id order -- the Jacobi tie
// rule, the block rule's lowest-id tie-break and the canonical triangle rank --
// is the single-image order shifted by a constant.  Then:
//   * the exact diagram's column and row pass run over all images at once, each
//     image kept within its own canvas, and one resolve over the atlas turns it
//     into the reference's fixed point (an explicit schedule, or what the resolve
//     leaves open, runs the passes over the atlas instead);
//   * one detection + dedup + numbering over the atlas; canonical global
//     ranks group by image (ids are contiguous per image), so an image's
//     triangle ids are the global ranks minus the count of earlier images';
//   * one set of tile lists over all triangles, each clipped to its own image with
//     its own image's degenerate-case window (per-image longest side);
//   * one launch draws every tile and writes the images' (H, W, 3) grids.
// The number of launches and host synchronisations is independent of the
// number of images.
#include "raster.cuh"
#include "exact_pass.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>
#include <numeric>
#include <string>
#include <vector>

namespace idl {
namespace {

constexpr int32_t WALL = (int32_t)0xFEFEFEFE;   // memset pattern 0xFE: below UNDEF

struct BImg {
    int W, H;          // image size
    int ox, oy;        // atlas origin of the padded canvas
    long long seed_off;  // first global seed id
    long long px_off;    // first output pixel (prefix of W*H); also the bitmap base
    int tile_off;        // first raster tile
    int tiles_x;         // raster tiles per row
};

// Image of each seed (ids of an image are contiguous, in input and in sorted
// order); a block per image.  Filled here: as host tables, these and the
// column and row tables below took 0.4 ms of a 512-image call to build and
// upload.
__global__ void k_b_seed_image(const BImg* __restrict__ imgs, int n_images, long long n, int32_t* __restrict__ seed_img)
{
    const int im = blockIdx.x;
    const long long end = im + 1 < n_images ? imgs[im + 1].seed_off : n;
    for (long long i = imgs[im].seed_off + threadIdx.x; i < end; i += blockDim.x) seed_img[i] = im;
}

__global__ void k_b_mark(const int32_t* __restrict__ xy, int64_t n, const int32_t* __restrict__ seed_img,
                         const BImg* __restrict__ imgs, uint32_t* __restrict__ bitmap,
                         unsigned long long* __restrict__ first_bad)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const BImg m = imgs[seed_img[i]];
    const int32_t x = xy[2 * i], y = xy[2 * i + 1];
    if (x < 0 || y < 0 || x >= m.W || y >= m.H) {
        atomicMin(&first_bad[0], (unsigned long long)i);
        return;
    }
    const long long bit = m.px_off + (long long)x * m.H + y;
    const uint32_t b = 1u << (bit & 31);
    if (atomicOr(&bitmap[bit >> 5], b) & b) atomicMin(&first_bad[1], (unsigned long long)i);
}

__global__ void k_b_rank(const int32_t* __restrict__ xy, int64_t n, const int32_t* __restrict__ seed_img,
                         const BImg* __restrict__ imgs, int P, const uint32_t* __restrict__ bitmap,
                         const int32_t* __restrict__ word_rank, int32_t* __restrict__ xs, int32_t* __restrict__ ys,
                         uint32_t* __restrict__ pos)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int im = seed_img[i];
    const BImg m = imgs[im];
    const int32_t x = xy[2 * i], y = xy[2 * i + 1];
    const long long bit = m.px_off + (long long)x * m.H + y;
    const int32_t r = word_rank[bit >> 5] + __popc(bitmap[bit >> 5] & ((1u << (bit & 31)) - 1u));
    xs[r] = x;
    ys[r] = y;
    pos[r] = pack_pos(m.ox + P + x, m.oy + P + y);
}

// Each image's padded canvas starts UNDEF (the rest of the atlas is WALL).
__global__ void k_b_open(int32_t* __restrict__ a, int32_t* __restrict__ b, int pitch, const BImg* __restrict__ imgs,
                         int P)
{
    const BImg m = imgs[blockIdx.y];
    const int Wp = m.W + 2 * P, Hp = m.H + 2 * P;
    for (int r = blockIdx.x; r < Hp; r += gridDim.x) {
        const size_t o = (size_t)(m.oy + r) * pitch + m.ox;
        for (int c = threadIdx.x; c < Wp; c += blockDim.x) {
            a[o + c] = UNDEF;
            b[o + c] = UNDEF;
        }
    }
}

__global__ void k_b_seeds(int32_t* __restrict__ a, int32_t* __restrict__ b, int pitch, const uint32_t* __restrict__ pos,
                          int64_t n)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t p = pos[i];
    const size_t o = (size_t)pos_y(p) * pitch + pos_x(p);
    a[o] = (int32_t)i;
    b[o] = (int32_t)i;
}

__device__ __forceinline__ int tri_image(const int32_t* row, const int32_t* __restrict__ sid_img)
{
    return sid_img[min(row[2], min(row[3], row[4]))];
}

// off[i] = first triangle of image i (off[n_images]: all of them).  Triangles
// are numbered by their smallest vertex and seeds image after image, so an
// image's triangles are contiguous: each boundary is written once, with no
// count per triangle (those atomics on a few hundred counters took 460 us for
// 1.2 M triangles of 512 images).
__global__ void k_b_tri_off(const int32_t* __restrict__ tris, const Scalars* __restrict__ sc,
                            const int32_t* __restrict__ sid_img, int n_images, int32_t* __restrict__ off)
{
    const long long nt = sc->n_triangles;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t <= nt;
         t += (long long)gridDim.x * blockDim.x) {
        const int im = t < nt ? tri_image(tris + t * 5, sid_img) : n_images;
        const int before = t > 0 ? tri_image(tris + (t - 1) * 5, sid_img) : -1;
        for (int i = before + 1; i <= im; ++i) off[i] = (int32_t)t;
    }
}

// The raster passes of raster.cu over the tiles of all images; the longest
// side is kept per image.
__global__ void __launch_bounds__(256)
k_b_raster_count(const int32_t* __restrict__ tris, const Scalars* __restrict__ sc,
                 const int32_t* __restrict__ sid_img, const BImg* __restrict__ imgs, const int32_t* __restrict__ xs,
                 const int32_t* __restrict__ ys, int32_t* __restrict__ side, RasterWork w)
{
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    const bool on = t < sc->n_triangles;
    Tri u{};
    int im = -1, side_here = 0, W = 0, H = 0, tile_off = 0, tiles_x = 0;
    if (on) {
        const int32_t* row = tris + t * 5;
        im = tri_image(row, sid_img);
        u = load_tri(row + 2, xs, ys);
        side_here = longest_side(u);
        W = imgs[im].W;
        H = imgs[im].H;
        tile_off = imgs[im].tile_off;
        tiles_x = imgs[im].tiles_x;
    }
    // a warp's triangles are mostly one image's: one atomic for all of them
    const int im0 = __shfl_sync(0xFFFFFFFFu, im, 0);
    if (__all_sync(0xFFFFFFFFu, im == im0 || im < 0)) {
        const int s = __reduce_max_sync(0xFFFFFFFFu, side_here);
        if ((threadIdx.x & 31) == 0 && im0 >= 0) atomicMax(&side[im0], s);
    } else if (on) {
        atomicMax(&side[im], side_here);
    }
    raster_count<TileLarge>(w, on, (int32_t)t, u, W, H, tile_off, tiles_x);
    raster_offsets<256>(w);
}

__global__ void __launch_bounds__(256)
k_b_raster_fill(const int32_t* __restrict__ tris, const Scalars* __restrict__ sc,
                const int32_t* __restrict__ sid_img, const BImg* __restrict__ imgs, RasterWork w)
{
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    if (w.head->overflow) return;
    const bool on = t < sc->n_triangles;
    const BImg& m = imgs[on ? tri_image(tris + t * 5, sid_img) : 0];
    raster_fill<TileLarge>(w, on, (int32_t)t, m.W, m.H, m.tile_off, m.tiles_x);
}

// A tile of its image drawn and composed: (local seed id, squared distance,
// triangle id) per pixel.
__global__ void __launch_bounds__(TILE_THREADS)
k_b_raster_compose(RasterWork w, const BImg* __restrict__ imgs, int n_images, const int32_t* __restrict__ tri_off,
                   const int32_t* __restrict__ lab, int pitch, int P, const int32_t* __restrict__ xs,
                   const int32_t* __restrict__ ys, int32_t* __restrict__ out)
{
    __shared__ int32_t pix[TileLarge::H * TileLarge::PITCH];
    int lo = 0, hi = n_images - 1;   // the last image whose first tile is at or before this one
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&imgs[mid].tile_off) <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const BImg m = imgs[lo];
    const int k = (int)blockIdx.x - m.tile_off, tx = k % m.tiles_x, ty = k / m.tiles_x;
    raster_tile<TileLarge>(w, pix, blockIdx.x, tx, ty, m.W, m.H, tri_off[lo]);
    compose_tile<TileLarge>(pix, tx, ty, m.W, m.H, lab + (size_t)(m.oy + P) * pitch + m.ox + P, pitch, xs, ys,
                 (int32_t)m.seed_off, out + m.px_off * 3);
}

__global__ void __launch_bounds__(128)
k_b_raster_rest(const int32_t* __restrict__ tris, const Scalars* __restrict__ sc,
                const int32_t* __restrict__ sid_img, const BImg* __restrict__ imgs, const int32_t* __restrict__ xs,
                const int32_t* __restrict__ ys, const int32_t* __restrict__ side,
                const int32_t* __restrict__ tri_off, int32_t* __restrict__ out, RasterWork w)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    const bool all = w.head->overflow != 0;
    const long long n = all ? sc->n_triangles : w.head->n_lines;
    for (long long i = warp; i < n; i += warps) {
        const int32_t t = all ? (int32_t)i : w.lines[i];
        const int32_t* row = tris + (size_t)t * 5;
        const int im = tri_image(row, sid_img);
        const BImg& m = imgs[im];
        const Tri u = load_tri(row + 2, xs, ys);
        int32_t* ids = out + m.px_off * 3 + 2;
        const int32_t id = t - tri_off[im];
        if (!u.line) raster_direct(u, ids, 3, m.W, m.H, id);
        else raster_line(u, ids, 3, m.W, m.H, id, max(20, side[im] + 3));
    }
}

// Triangle rows to image-local form: witness relative to the image (shifted
// by -P as the single-image path reports it), vertex ids local.
__global__ void k_b_localise(int32_t* __restrict__ tris, const Scalars* __restrict__ sc,
                             const int32_t* __restrict__ sid_img, const BImg* __restrict__ imgs, int P)
{
    const long long nt = sc->n_triangles;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nt;
         t += (long long)gridDim.x * blockDim.x) {
        int32_t* row = tris + t * 5;
        const BImg m = imgs[tri_image(row, sid_img)];
        row[0] -= m.ox + P;
        row[1] -= m.oy + P;
        row[2] = (int32_t)(row[2] - m.seed_off);
        row[3] = (int32_t)(row[3] - m.seed_off);
        row[4] = (int32_t)(row[4] - m.seed_off);
    }
}

inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

struct Plan {
    std::vector<BImg> imgs;
    int AW = 0, AH = 0;
    int64_t n_seeds = 0, n_px = 0, n_tiles = 0;
};

// Shelf packing of the padded canvases, tallest first, one wall cell apart.
Plan make_plan(int n_images, const int32_t* dims, const int64_t* counts, int P)
{
    if (n_images <= 0) invalid("a batch needs at least one image");
    if (n_images > 65535) invalid("at most 65535 images per batch are supported");
    Plan pl;
    pl.imgs.resize(n_images);
    double area = 0;
    int max_wp = 0;
    for (int i = 0; i < n_images; ++i) {
        const int W = dims[2 * i], H = dims[2 * i + 1];
        const int64_t n = counts[i];
        if (W <= 0 || H <= 0) {
            if (n <= 0) invalid("image " + std::to_string(i) + ": seeds must not be empty");
            invalid("image " + std::to_string(i) + ": seed coordinate out of bounds");
        }
        if (n <= 0) invalid("image " + std::to_string(i) + ": seeds must not be empty");
        if ((int64_t)W + 2 * P + 1 > MAX_CANVAS_SIDE || (int64_t)H + 2 * P + 1 > MAX_CANVAS_SIDE)
            invalid("image " + std::to_string(i) + ": canvas side (including border padding) must not exceed " +
                    std::to_string(MAX_CANVAS_SIDE - 1));
        BImg& m = pl.imgs[i];
        m.W = W;
        m.H = H;
        m.seed_off = pl.n_seeds;
        m.px_off = pl.n_px;
        pl.n_seeds += n;
        pl.n_px += (int64_t)W * H;
        m.tile_off = (int)pl.n_tiles;
        m.tiles_x = ceil_div(W, TileLarge::W);
        pl.n_tiles += (int64_t)m.tiles_x * ceil_div(H, TileLarge::H);
        area += (double)(W + 2 * P + 1) * (H + 2 * P + 1);
        max_wp = std::max(max_wp, W + 2 * P + 1);
    }
    if (pl.n_seeds > MAX_SEEDS) invalid("at most " + std::to_string(MAX_SEEDS) + " seeds per batch are supported");
    std::vector<int> order(n_images);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return pl.imgs[a].H > pl.imgs[b].H; });
    int AW = std::max(max_wp, (int)std::ceil(std::sqrt(area) * 1.05));
    AW = std::min(MAX_CANVAS_SIDE, (AW + 31) / 32 * 32);
    int x = 0, y = 0, shelf = 0;
    for (int i : order) {
        BImg& m = pl.imgs[i];
        const int wp = m.W + 2 * P + 1, hp = m.H + 2 * P + 1;
        if (x + wp > AW) {
            y += shelf;
            x = 0;
            shelf = 0;
        }
        m.ox = x;
        m.oy = y;
        x += wp;
        shelf = std::max(shelf, hp);
    }
    const int64_t AH = (int64_t)y + shelf;
    if (AH > MAX_CANVAS_SIDE) invalid("batch too large for one atlas: split it into smaller batches");
    pl.AW = AW;
    pl.AH = (int)AH;
    return pl;
}

// The pipeline; seeds already in C.seeds_in.  Leaves per-image grids in
// d_out (or C.outgrid) and image-local triangle rows in C.tris.
// What idl_delaunay_adopt (and batch_fetch) need of the last batch on a
// context: the atlas layout, and after the whole pipeline, where each
// image's grid and triangle rows are.
struct BatchPlan {
    std::vector<BImg> imgs;
    int P = 0, pitch = 0;
    int64_t n_seeds = 0;
    bool full = false;               // grids in `grids`, image-local rows in C.tris
    bool exact = false;              // labels of the exact semantics (not adoptable)
    const int32_t* grids = nullptr;  // device, n_px x 3 int32
    std::vector<int64_t> tri_off;    // n_images + 1 row offsets
};

// Exact-semantics labels of every image into C.lab[0] (the atlas's walls
// stay) by the passes of exact.cu, each image kept within its own canvas: a
// column walk uses only its image's seeds, a row only its image's columns, so
// no label crosses a wall.  Labels are global seed ids, as the Jacobi path
// leaves them; the column pass's plane is in C.lab[1].  Returns the image
// table on the device.
const XImg* exact_atlas(Context& C, const Plan& pl, int P, const Canvas& cv)
{
    const int n_images = (int)pl.imgs.size();
    std::vector<XImg> xi(n_images);
    int n_pairs = 0, n_rows = 0;
    int max_wp = 0, max_hp = 0;
    int64_t band_entries = 0;
    for (int i = 0; i < n_images; ++i) {
        const BImg& b = pl.imgs[i];
        XImg& m = xi[i];
        m.ox = b.ox;
        m.oy = b.oy;
        m.Wp = b.W + 2 * P;
        m.Hp = b.H + 2 * P;
        m.pair_off = n_pairs;
        m.row_off = n_rows;
        m.band_off = (int)band_entries;
        m.s0 = (int)b.seed_off;
        m.s1 = (int)(i + 1 < n_images ? pl.imgs[i + 1].seed_off : pl.n_seeds);
        n_pairs += (m.Wp + 1) / 2;
        n_rows += m.Hp;
        band_entries += (int64_t)x_bands(m) * m.Wp;
        m.P = P;
        m.bit0 = b.px_off;
        max_wp = std::max(max_wp, m.Wp);
        max_hp = std::max(max_hp, m.Hp);
    }
    C.batch_ximg.ensure(xi.size() * sizeof(XImg));
    C.batch_colimg.ensure((size_t)n_pairs * 4);
    C.batch_rowimg.ensure((size_t)n_rows * 4);
    IDL_CUDA(cudaMemcpyAsync(C.batch_ximg.ptr, xi.data(), xi.size() * sizeof(XImg), cudaMemcpyHostToDevice,
                             C.stream));
    const XImg* d_xi = C.batch_ximg.as<XImg>();
    exact_images(C, cv.pitch, C.pos.as<uint32_t>(), d_xi, n_images, C.batch_colimg.as<int32_t>(), n_pairs,
                 C.batch_rowimg.as<int32_t>(), n_rows, max_wp, max_hp, band_entries);
    return d_xi;
}

void run_batch(Context& C, const Plan& pl, int P, int n_images, int32_t* d_out, int64_t* tri_counts,
               float* timings, bool labels_only = false, int mode = IDL_MODE_REFERENCE)
{
    C.batch_plan.reset();
    C.owner = nullptr;
    const int64_t n = pl.n_seeds;
    C.batch_img.ensure(pl.imgs.size() * sizeof(BImg));
    C.batch_seed_img.ensure((size_t)n * 4);
    C.batch_stats.ensure(((size_t)n_images * 2 + 1) * 4);
    BImg* d_imgs = C.batch_img.as<BImg>();
    IDL_CUDA(cudaMemcpyAsync(d_imgs, pl.imgs.data(), pl.imgs.size() * sizeof(BImg), cudaMemcpyHostToDevice,
                             C.stream));
    k_b_seed_image<<<(unsigned)n_images, 256, 0, C.stream>>>(d_imgs, n_images, n, C.batch_seed_img.as<int32_t>());
    IDL_LAUNCH();
    cudaEvent_t ev[5] = {};
    if (timings)
        for (auto& e : ev) IDL_CUDA(cudaEventCreate(&e));
    struct Ev {
        cudaEvent_t* e;
        ~Ev()
        {
            for (int i = 0; i < 5; ++i)
                if (e[i]) cudaEventDestroy(e[i]);
        }
    } ev_guard{ev};
    auto mark = [&](int i) {
        if (timings) IDL_CUDA(cudaEventRecord(ev[i], C.stream));
    };

    // validate + rank
    const int64_t nwords = (pl.n_px + 31) / 32;
    C.bitmap.ensure((size_t)nwords * 4);
    C.scan_c.ensure((size_t)(nwords + 1) * 4);
    C.xs.ensure((size_t)n * 4);
    C.ys.ensure((size_t)n * 4);
    C.pos.ensure((size_t)n * 4);
    C.batch_bad.ensure(16);
    unsigned long long* bad = C.batch_bad.as<unsigned long long>();
    ClearList zero;
    zero.add(C.bitmap.ptr, (size_t)nwords * 4, 0);
    zero.add(bad, 16, 0xFFFFFFFFu);
    zero.add(reinterpret_cast<char*>(C.sc()) + SCAN_UNIT, 16, 0);
    clear_buffers(C, zero);
    mark(0);
    k_b_mark<<<nblk(n), 256, 0, C.stream>>>(C.seeds_in.as<int32_t>(), n, C.batch_seed_img.as<int32_t>(), d_imgs,
                                           C.bitmap.as<uint32_t>(), bad);
    IDL_LAUNCH();
    unsigned long long hb[2] = {0, 0};
    IDL_CUDA(cudaMemcpyAsync(hb, bad, 16, cudaMemcpyDeviceToHost, C.stream));
    IDL_CUDA(cudaStreamSynchronize(C.stream));
    auto image_of = [&](unsigned long long i) {
        return (int)(std::upper_bound(pl.imgs.begin(), pl.imgs.end(), (long long)i,
                                      [](long long v, const BImg& m) { return v < m.seed_off; }) -
                     pl.imgs.begin()) - 1;
    };
    if (hb[0] != ~0ull) invalid("image " + std::to_string(image_of(hb[0])) + ": seed coordinate out of bounds");
    if (hb[1] != ~0ull)
        invalid("image " + std::to_string(image_of(hb[1])) + ": duplicate seed positions are not allowed");
    exclusive_popc_scan(C, C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), nwords);
    k_b_rank<<<nblk(n), 256, 0, C.stream>>>(C.seeds_in.as<int32_t>(), n, C.batch_seed_img.as<int32_t>(), d_imgs, P,
                                           C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), C.xs.as<int32_t>(),
                                           C.ys.as<int32_t>(), C.pos.as<uint32_t>());
    IDL_LAUNCH();

    const Canvas cv{pl.AW, pl.AH, (pl.AW + 31) / 32 * 32};
    const size_t plane = (size_t)cv.pitch * cv.Hd * 4;
    C.lab[0].ensure(plane);
    C.lab[1].ensure(plane);
    mark(1);
    auto run_passes = [&] {
        // atlas planes: walls everywhere, each image's padded canvas open, seeds in
        IDL_CUDA(cudaMemsetAsync(C.lab[0].ptr, 0xFE, plane, C.stream));
        IDL_CUDA(cudaMemsetAsync(C.lab[1].ptr, 0xFE, plane, C.stream));
        k_b_open<<<dim3(64, n_images), 256, 0, C.stream>>>(C.lab[0].as<int32_t>(), C.lab[1].as<int32_t>(), cv.pitch,
                                                           d_imgs, P);
        IDL_LAUNCH();
        k_b_seeds<<<nblk(n), 256, 0, C.stream>>>(C.lab[0].as<int32_t>(), C.lab[1].as<int32_t>(), cv.pitch,
                                                C.pos.as<uint32_t>(), n);
        IDL_LAUNCH();
        propagate(C, IDL_MODE_REFERENCE, cv, C.pos.as<uint32_t>(), n);
    };
    const bool direct = mode == IDL_MODE_REFERENCE && C.direct();
    if (mode == IDL_MODE_EXACT || direct) {
        // the exact passes write every cell of every image; the walls between
        // them are read by the block rule (and by resolve_exact) in plane 0 only
        IDL_CUDA(cudaMemsetAsync(C.lab[0].ptr, 0xFE, plane, C.stream));
        const XImg* xi = exact_atlas(C, pl, P, cv);
        if (direct) resolve_exact(C, cv, C.pos.as<uint32_t>(), n, xi, C.batch_seed_img.as<int32_t>());
    } else {
        run_passes();
    }
    mark(2);
    auto bp = std::make_shared<BatchPlan>();
    bp->imgs = pl.imgs;
    bp->P = P;
    bp->pitch = cv.pitch;
    bp->n_seeds = n;
    bp->exact = mode == IDL_MODE_EXACT;
    C.batch_plan = bp;
    if (labels_only) {
        if (direct) {
            C.fetch_scalars();
            if (!resolved(C)) run_passes();
        }
        return;
    }
    detect_triangles(C, cv, C.lab[0].as<int32_t>(), C.pos.as<uint32_t>(), n, 0, timings ? ev[3] : nullptr);
    if (direct && !resolved(C)) {
        // the exact diagram did not decide some image's fixed point: run the passes
        run_passes();
        mark(2);
        detect_triangles(C, cv, C.lab[0].as<int32_t>(), C.pos.as<uint32_t>(), n, 0, timings ? ev[3] : nullptr);
    }

    // per-image counts, offsets and windows; raster; compose
    int32_t* side = C.batch_stats.as<int32_t>();
    int32_t* off = side + n_images;   // n_images + 1
    const int64_t nt = C.host_sc->n_triangles;
    IDL_CUDA(cudaMemsetAsync(side, 0, (size_t)n_images * 4, C.stream));
    k_b_tri_off<<<nblk(nt + 1), 256, 0, C.stream>>>(C.tris.as<int32_t>(), C.sc(), C.batch_seed_img.as<int32_t>(), n_images,
                                                   off);
    IDL_LAUNCH();
    int32_t* out = d_out;
    if (!out) {
        C.outgrid.ensure((size_t)pl.n_px * 12);
        out = C.outgrid.as<int32_t>();
    }
    const RasterWork w = raster_work(C, nt, pl.n_tiles);
    const int32_t* sid = C.batch_seed_img.as<int32_t>();
    const int32_t *xs = C.xs.as<int32_t>(), *ys = C.ys.as<int32_t>(), *tris = C.tris.as<int32_t>();
    if (nt > 0) {
        k_b_raster_count<<<nblk(nt), 256, 0, C.stream>>>(tris, C.sc(), sid, d_imgs, xs, ys, side, w);
        IDL_LAUNCH();
        k_b_raster_fill<<<nblk(nt), 256, 0, C.stream>>>(tris, C.sc(), sid, d_imgs, w);
        IDL_LAUNCH();
    } else {
        IDL_CUDA(cudaMemsetAsync(w.off, 0, ((size_t)pl.n_tiles + 1) * 4, C.stream));
    }
    k_b_raster_compose<<<(unsigned)pl.n_tiles, TILE_THREADS, 0, C.stream>>>(w, d_imgs, n_images, off,
                                                                          C.lab[0].as<int32_t>(), cv.pitch, P, xs, ys,
                                                                          out);
    IDL_LAUNCH();
    if (nt > 0) {
        k_b_raster_rest<<<C.num_sms, 128, 0, C.stream>>>(tris, C.sc(), sid, d_imgs, xs, ys, side, off, out, w);
        IDL_LAUNCH();
    }
    k_b_localise<<<C.num_sms * 8, 256, 0, C.stream>>>(C.tris.as<int32_t>(), C.sc(), C.batch_seed_img.as<int32_t>(),
                                                      d_imgs, P);
    IDL_LAUNCH();
    mark(4);
    std::vector<int32_t> ho((size_t)n_images + 1);
    IDL_CUDA(cudaMemcpyAsync(ho.data(), off, ho.size() * 4, cudaMemcpyDeviceToHost, C.stream));
    C.fetch_scalars();
    C.last_n_tri = C.host_sc->n_triangles;
    C.have_result = true;
    if (tri_counts)
        for (int i = 0; i < n_images; ++i) tri_counts[i] = ho[i + 1] - ho[i];
    bp->tri_off.assign(ho.begin(), ho.end());
    bp->grids = out;
    bp->full = true;
    if (timings) {
        float a = 0, b = 0, c = 0, d = 0;
        IDL_CUDA(cudaEventElapsedTime(&a, ev[1], ev[2]));
        IDL_CUDA(cudaEventElapsedTime(&b, ev[2], ev[3]));
        IDL_CUDA(cudaEventElapsedTime(&c, ev[3], ev[4]));
        IDL_CUDA(cudaEventElapsedTime(&d, ev[0], ev[1]));
        timings[IDL_T_BFS_MS] = a;
        timings[IDL_T_DETECT_MS] = b;
        timings[IDL_T_DEDUP_MS] = 0.f;
        timings[IDL_T_ASSIGN_MS] = c;
        timings[IDL_T_BFS_ITERS] = 0.f;
        (void)d;
    }
}

}  // namespace

void triangulate_batch_keep(Context& C, int n_images, const int32_t* dims, const int64_t* counts,
                            const int32_t* seeds_xy, int P, int64_t* tri_counts)
{
    if (!dims || !counts) invalid("dims and seed_counts must not be NULL");
    const Plan pl = make_plan(n_images, dims, counts, P);
    if (!seeds_xy) invalid("seeds must not be NULL");
    DeviceGuard g(C.device);
    C.have_result = false;
    C.batch_plan.reset();
    C.seeds_in.ensure((size_t)pl.n_seeds * 8);
    IDL_CUDA(cudaMemcpyAsync(C.seeds_in.ptr, seeds_xy, (size_t)pl.n_seeds * 8, cudaMemcpyHostToDevice, C.stream));
    run_batch(C, pl, P, n_images, nullptr, tri_counts, nullptr);
}

void batch_fetch(Context& C, int k, int32_t* grid_out, int32_t* tris_out, int64_t capacity)
{
    const auto* bp = static_cast<const BatchPlan*>(C.batch_plan.get());
    if (!bp || !bp->full || k < 0 || k >= (int)bp->imgs.size())
        throw Error(IDL_ERR_STATE, "no triangulated batch image " + std::to_string(k) + " on this context");
    const BImg& m = bp->imgs[k];
    if (grid_out)
        IDL_CUDA(cudaMemcpyAsync(grid_out, bp->grids + (size_t)m.px_off * 3, (size_t)m.W * m.H * 12,
                                 cudaMemcpyDeviceToHost, C.stream));
    const int64_t rows = bp->tri_off[k + 1] - bp->tri_off[k];
    if (tris_out && rows) {
        if (capacity < rows * 5) invalid("triangle buffer too small");
        IDL_CUDA(cudaMemcpyAsync(tris_out, C.tris.as<int32_t>() + bp->tri_off[k] * 5, (size_t)rows * 20,
                                 cudaMemcpyDeviceToHost, C.stream));
    }
}

bool batch_image(const Context& C, int k, BatchImage& out)
{
    const auto* lo = static_cast<const BatchPlan*>(C.batch_plan.get());
    if (!lo || lo->exact || k < 0 || k >= (int)lo->imgs.size()) return false;
    const BImg& m = lo->imgs[k];
    out.W = m.W;
    out.H = m.H;
    out.ox = m.ox;
    out.oy = m.oy;
    out.P = lo->P;
    out.pitch = lo->pitch;
    out.seed_off = m.seed_off;
    out.n = (k + 1 < (int)lo->imgs.size() ? lo->imgs[k + 1].seed_off : lo->n_seeds) - m.seed_off;
    return true;
}

}  // namespace idl

using namespace idl;

extern "C" {

int idl_voronoi_batch(idl_context* ctx, int n_images, const int32_t* dims, const int64_t* seed_counts,
                      const int32_t* seeds_xy, int border_padding, int mode)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (!dims || !seed_counts) invalid("dims and seed_counts must not be NULL");
    if (mode != IDL_MODE_REFERENCE) invalid("batched propagation supports voronoi_mode 'reference' only");
    const int P = border_padding == IDL_AUTO_BORDER_PADDING ? IDL_DEFAULT_BORDER_PADDING
                                                            : std::max(0, border_padding);
    const Plan pl = make_plan(n_images, dims, seed_counts, P);
    if (!seeds_xy) invalid("seeds must not be NULL");
    DeviceGuard g(ctx->device);
    Context& C = *ctx;
    C.have_result = false;
    C.batch_plan.reset();
    C.seeds_in.ensure((size_t)pl.n_seeds * 8);
    IDL_CUDA(cudaMemcpyAsync(C.seeds_in.ptr, seeds_xy, (size_t)pl.n_seeds * 8, cudaMemcpyHostToDevice, C.stream));
    run_batch(C, pl, P, n_images, nullptr, nullptr, nullptr, true);
    IDL_API_END
}

int idl_triangulate_batch(idl_context* ctx, int n_images, const int32_t* dims, const int64_t* seed_counts,
                          const int32_t* seeds_xy, int border_padding, int mode, int32_t* grids_out,
                          int64_t* tri_counts_out, float* timings_out)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (!dims || !seed_counts) invalid("dims and seed_counts must not be NULL");
    if (mode != IDL_MODE_REFERENCE && mode != IDL_MODE_EXACT)
        invalid("batched triangulation supports voronoi_mode 'reference' and 'exact'");
    const int P = border_padding == IDL_AUTO_BORDER_PADDING ? IDL_DEFAULT_BORDER_PADDING
                                                            : std::max(0, border_padding);
    const Plan pl = make_plan(n_images, dims, seed_counts, P);
    if (!seeds_xy) invalid("seeds must not be NULL");
    DeviceGuard g(ctx->device);
    Context& C = *ctx;
    C.have_result = false;
    C.seeds_in.ensure((size_t)pl.n_seeds * 8);
    IDL_CUDA(cudaMemcpyAsync(C.seeds_in.ptr, seeds_xy, (size_t)pl.n_seeds * 8, cudaMemcpyHostToDevice, C.stream));
    run_batch(C, pl, P, n_images, nullptr, tri_counts_out, timings_out, false, mode);
    if (grids_out)
        IDL_CUDA(cudaMemcpyAsync(grids_out, C.outgrid.ptr, (size_t)pl.n_px * 12, cudaMemcpyDeviceToHost, C.stream));
    IDL_CUDA(cudaStreamSynchronize(C.stream));
    IDL_API_END
}

int idl_triangulate_batch_device(idl_context* ctx, int n_images, const int32_t* dims, const int64_t* seed_counts,
                                 const int32_t* d_seeds_xy, int border_padding, int mode, int32_t* d_grids_out,
                                 int64_t* tri_counts_out)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (!dims || !seed_counts) invalid("dims and seed_counts must not be NULL");
    if (mode != IDL_MODE_REFERENCE && mode != IDL_MODE_EXACT)
        invalid("batched triangulation supports voronoi_mode 'reference' and 'exact'");
    const int P = border_padding == IDL_AUTO_BORDER_PADDING ? IDL_DEFAULT_BORDER_PADDING
                                                            : std::max(0, border_padding);
    const Plan pl = make_plan(n_images, dims, seed_counts, P);
    if (!d_seeds_xy || !d_grids_out) invalid("device buffers must not be NULL");
    DeviceGuard g(ctx->device);
    Context& C = *ctx;
    C.have_result = false;
    C.seeds_in.ensure((size_t)pl.n_seeds * 8);
    IDL_CUDA(cudaMemcpyAsync(C.seeds_in.ptr, d_seeds_xy, (size_t)pl.n_seeds * 8, cudaMemcpyDeviceToDevice,
                             C.stream));
    run_batch(C, pl, P, n_images, d_grids_out, tri_counts_out, nullptr, false, mode);
    IDL_API_END
}

}  // extern "C"
