// Stage (d): which triangle contains each pixel.
//
// Reference semantics (src/cuda/triangulation.cu:101-137 with
// geometry_device.cuh:68-86): pixel (x, y) is the integer point (x, y); it
// belongs to the highest triangle id among the detected triangles whose closed
// point-in-triangle test accepts it, and to -1 if none does.  The reference
// finds candidates by looping over ALL seeds per pixel, keeping those within a
// Chebyshev window_cap = max(20, max_side + 3) (max_side: the longest side over
// all triangles, float-truncated, triangulation.cu:355-368), and testing their
// CSR triangles -- O(W*H*N) work.
//
// Here each triangle rasterises itself instead: for every row its vertices
// span, the exact integer x-interval of the closed triangle is found from the
// three edge functions in integers, and atomicMax writes the triangle id into
// every pixel of it.  The window never excludes a pixel of a non-degenerate
// triangle (any vertex of a triangle is within its longest side of every
// point inside it, and window_cap exceeds every side), so the result is the
// same set union, computed in O(covered pixels).
//
// Two details keep it bit-equal:
//  * The reference's test is float.  For pixel and seed coordinates in
//    [0, 4096) every product in it is an exact float below 2^24 and the sign
//    of the difference is exact, so float and integers agree; beyond that the
//    integer test is the exact one.
//  * A degenerate (collinear) triangle passes the closed test at every point
//    of its supporting line (all three cross products are 0) and nowhere else.
//    The reference then reaches it only through the window, so such a triangle
//    covers the points of its line within Chebyshev window_cap of one of its
//    vertices, clipped to the image.  That case is rasterised separately.
#include "raster.cuh"

namespace idl {
namespace {

// Triangles of one image to the lanes of the list kernels: `per` lanes of every
// warp, eight consecutive triangles at a time, so that the large triangles around
// one seed, consecutive by their numbers, fall to many warps (a disc of 84 000
// seeds and five far ones, an atomic each: 72 + 91 us with 32 consecutive ones to
// a warp, 56 + 53 with eight, 47 + 46 with four).  Eight rows, and eight triangles' corners, are
// whole 32-byte sectors; with four, 200 000 uniform seeds took 2 to 10 us more,
// by the device.
constexpr int LEAST = 4, CHUNK = 8;

__device__ __forceinline__ long long triangle_of_lane(int per)
{
    const int lane = threadIdx.x & 31, chunk = per < CHUNK ? per : CHUNK;
    const long long warps = (long long)gridDim.x * 8, warp = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    return lane < per ? (lane / CHUNK * warps + warp) * chunk + lane % CHUNK : 0x7FFFFFFFFFFFFFFFll;
}

// Triangles to draw: none if there is no room for all of them, since the caller
// then draws them again.
__device__ __forceinline__ long long drawn(const Scalars* sc, const RasterWork& w)
{
    const long long nt = sc->n_triangles;
    return nt <= w.max_tri ? nt : 0;
}

template <class TILE>
__global__ void __launch_bounds__(256)
k_raster_count(const int32_t* __restrict__ tris, Scalars* __restrict__ sc, const int32_t* __restrict__ xs,
               const int32_t* __restrict__ ys, int W, int H, RasterWork w, int per)
{
    const int tiles_x = (W + TILE::W - 1) / TILE::W;
    const long long t = triangle_of_lane(per);
    const bool on = t < drawn(sc, w);
    Tri u{};
    if (on) u = load_tri(tris + t * 5 + 2, xs, ys);
    int side = on ? longest_side(u) : 0;
    raster_count<TILE>(w, on, (int32_t)t, u, W, H, 0, tiles_x);
    side = __reduce_max_sync(0xFFFFFFFFu, side);
    if ((threadIdx.x & 31) == 0 && side > __ldcg(&w.head->max_side)) atomicMax(&w.head->max_side, side);
    raster_offsets<256>(w);
}

template <class TILE>
__global__ void __launch_bounds__(256)
k_raster_fill(const Scalars* __restrict__ sc, int W, int H, RasterWork w, int per)
{
    const long long t = triangle_of_lane(per);
    if (!w.head->overflow)
        raster_fill<TILE>(w, t < drawn(sc, w), (int32_t)t, W, H, 0, (W + TILE::W - 1) / TILE::W);
}

template <class TILE>
__global__ void __launch_bounds__(TILE_THREADS)
k_raster_tiles(RasterWork w, int W, int H, int32_t* __restrict__ tgrid)
{
    __shared__ int32_t pix[TILE::H * TILE::PITCH];
    const int tiles_x = (W + TILE::W - 1) / TILE::W;
    const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
    raster_tile<TILE>(w, pix, blockIdx.x, tx, ty, W, H, 0);
    const int x = tx * TILE::W + (threadIdx.x % TILE::W);
    if (x >= W) return;
    for (int r = threadIdx.x / TILE::W; r < TILE::H && ty * TILE::H + r < H; r += TILE_THREADS / TILE::W)
        tgrid[(size_t)(ty * TILE::H + r) * W + x] = pix[r * TILE::PITCH + threadIdx.x % TILE::W];
}

// The same with the (H, W, 3) output composed on the way out, so that the
// triangle ids never go through memory on their own.
template <class TILE>
__global__ void __launch_bounds__(TILE_THREADS)
k_raster_compose(RasterWork w, int W, int H, const int32_t* __restrict__ lab, int pitch,
                 const int32_t* __restrict__ xs, const int32_t* __restrict__ ys, int32_t* __restrict__ out)
{
    __shared__ int32_t pix[TILE::H * TILE::PITCH];
    const int tiles_x = (W + TILE::W - 1) / TILE::W;
    const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
    raster_tile<TILE>(w, pix, blockIdx.x, tx, ty, W, H, 0);
    compose_tile<TILE>(pix, tx, ty, W, H, lab, pitch, xs, ys, 0, out);
}

// The collinear triangles (the longest side is known by now), and all of them
// if the tile lists did not fit.
__global__ void __launch_bounds__(128)
k_raster_rest(const int32_t* __restrict__ tris, const Scalars* __restrict__ sc, const int32_t* __restrict__ xs,
              const int32_t* __restrict__ ys, int W, int H, int32_t* __restrict__ tgrid, int stride, RasterWork w)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    if (w.head->overflow)
        for (long long t = warp; t < sc->n_triangles; t += warps) {
            const Tri u = load_tri(tris + t * 5 + 2, xs, ys);
            if (!u.line) raster_direct(u, tgrid, stride, W, H, (int32_t)t);
        }
    const int n = w.head->n_lines;
    for (int i = warp; i < n; i += warps) {
        const int32_t t = w.lines[i];
        raster_line(load_tri(tris + (size_t)t * 5 + 2, xs, ys), tgrid, stride, W, H, t, max(20, w.head->max_side + 3));
    }
}

}  // namespace

namespace {

constexpr size_t HEAD_BYTES = 256;

// At 200 000 uniform seeds a triangle meets 1.6 tiles.  Where they are long
// slivers, it is the tile that bounds them: those that cross it do not overlap,
// so they are about as many as its rows and columns, here 96, however many tiles
// each of them meets (seeds on two opposite sides of the image; without the
// second term their lists did not fit and every pixel was an atomic in memory:
// 261 us at 2048 x 2048).  Triangles of a caller's grid may overlap and need more; those go straight
// into the image.
int64_t list_capacity(const Context& C, int64_t nt, int64_t n_tiles)
{
    return C.selftest.bound(IDL_LIMIT_TILE_LISTS,
                            std::min<int64_t>(4 * nt + 128 * n_tiles + 65536, (int64_t)1 << 30));
}

size_t work_reserve(Context& C, int64_t nt, int64_t n_tiles)
{
    C.rbig.ensure(HEAD_BYTES + ((size_t)n_tiles * 2 + 1 + (size_t)nt * 4 + (size_t)list_capacity(C, nt, n_tiles)) * 4);
    return HEAD_BYTES + (size_t)n_tiles * 4;
}

template <class TILE>
int64_t tile_count(int W, int H) { return (int64_t)ceil_div(W, TILE::W) * ceil_div(H, TILE::H); }

}  // namespace

size_t raster_reserve(Context& C, int W, int H, int64_t n_tri)
{
    const int64_t large = tile_count<TileLarge>(W, H);
    return work_reserve(C, n_tri, small_tiles(large, C.num_sms) ? tile_count<TileSmall>(W, H) : large);
}

RasterWork raster_work(Context& C, int64_t nt, int64_t n_tiles)
{
    const size_t zero = work_reserve(C, nt, n_tiles);
    char* base = C.rbig.as<char>();
    RasterWork w;
    w.head = reinterpret_cast<RasterHead*>(base);
    w.count = reinterpret_cast<int32_t*>(base + HEAD_BYTES);
    w.off = w.count + n_tiles;
    w.lines = w.off + n_tiles + 1;
    w.xy = reinterpret_cast<uint32_t*>(w.lines + nt);
    w.list = reinterpret_cast<int32_t*>(w.xy + nt * 3);
    w.n_tiles = (int32_t)n_tiles;
    w.list_cap = (int32_t)list_capacity(C, nt, n_tiles);
    w.max_tri = (int32_t)nt;
    if (!C.precleared) IDL_CUDA(cudaMemsetAsync(base, 0, zero, C.stream));
    return w;
}

namespace {

// Tile lists of the triangles in C.tris, then draw(tile, tiles, work) and the
// rest pass on the pixel ids at `ids`, `stride` ints apart.
template <class TILE, class F>
void raster_with(Context& C, int W, int H, const int32_t* xs, const int32_t* ys, int64_t n_tri, int32_t* ids,
                 int stride, bool overlap, F&& draw)
{
    const int64_t tiles = tile_count<TILE>(W, H);
    const RasterWork w = raster_work(C, n_tri, tiles);
    const int32_t* tris = C.tris.as<int32_t>();
    if (n_tri > 0) {
        // few triangles: fewer to a warp, so that every SM has some
        int per = 32;
        while (per > LEAST && n_tri < (int64_t)C.num_sms * 8 * per) per /= 2;
        const unsigned blocks = (unsigned)ceil_div(n_tri, 8 * per);
        k_raster_count<TILE><<<blocks, 256, 0, C.stream>>>(tris, C.sc(), xs, ys, W, H, w, per);
        IDL_LAUNCH();
        k_raster_fill<TILE><<<blocks, 256, 0, C.stream>>>(C.sc(), W, H, w, per);
        IDL_LAUNCH();
    } else {
        IDL_CUDA(cudaMemsetAsync(w.off, 0, ((size_t)tiles + 1) * 4, C.stream));
    }
    draw(TILE{}, (unsigned)tiles, w);
    IDL_LAUNCH();
    if (n_tri > 0) {
        // 16 blocks per SM where the lists may not fit (218 us for 8 000 random
        // triangles across 512 x 512, 696 with one), one where they do: it finds
        // next to nothing to draw
        k_raster_rest<<<C.num_sms * (overlap ? 16 : 1), 128, 0, C.stream>>>(tris, C.sc(), xs, ys, W, H, ids, stride, w);
        IDL_LAUNCH();
    }
}

template <class F>
void raster(Context& C, int W, int H, const int32_t* xs, const int32_t* ys, int64_t n_tri, int32_t* ids, int stride,
            bool overlap, F&& draw)
{
    if (small_tiles(tile_count<TileLarge>(W, H), C.num_sms))
        raster_with<TileSmall>(C, W, H, xs, ys, n_tri, ids, stride, overlap, draw);
    else raster_with<TileLarge>(C, W, H, xs, ys, n_tri, ids, stride, overlap, draw);
}

}  // namespace

void assign_pixels(Context& C, int W, int H, const int32_t* xs, const int32_t* ys, int32_t* tgrid, int64_t n_tri,
                   bool overlap)
{
    raster(C, W, H, xs, ys, n_tri, tgrid, 1, overlap, [&](auto tile, unsigned tiles, const RasterWork& w) {
        k_raster_tiles<decltype(tile)><<<tiles, TILE_THREADS, 0, C.stream>>>(w, W, H, tgrid);
    });
}

void assign_and_compose(Context& C, int W, int H, const int32_t* xs, const int32_t* ys, int64_t n_tri,
                        const int32_t* lab, int pitch, int32_t* out)
{
    raster(C, W, H, xs, ys, n_tri, out + 2, 3, false, [&](auto tile, unsigned tiles, const RasterWork& w) {
        k_raster_compose<decltype(tile)><<<tiles, TILE_THREADS, 0, C.stream>>>(w, W, H, lab, pitch, xs, ys, out);
    });
}

}  // namespace idl
