// Stage (a), exact semantics (IDL_MODE_EXACT): every cell takes the nearest
// seed in squared L2 distance, ties to the higher seed id -- the contract the
// reference's two implementations approximate (src/delauney/reference/
// voronoi.py:9-31; its NumPy sweep meets it on every probe, its CUDA Jacobi
// iteration misses a few "orphan" cells).  The result depends only on the
// seed set, not on any propagation history.
//
// Separable and exact, in two data-parallel passes over the canvas
// (exact_pass.cuh): the nearest seed of each cell's own column, then each
// cell's best over its row's column candidates, by winners that only move
// right along the row.
// Completeness: the nearest seed s* of a cell lies in some column x*, whose
// column candidate is at least as near (and, if as near, is the higher-id
// one of the two equidistant seeds in that column); two candidates from
// different columns at equal distance are ordered by column, i.e. by id.
// Seed ids are (x asc, y asc) ranks, so "higher id" is a comparison of ids.
//
// Measured at 4096 x 4096 / 200 000 uniform seeds (B200): column pass 31 us
// (two bytes per cell and a table entry per 64 written, 57 % issue), row pass
// 129 us (bound by instruction issue: 85 % of cycles); with a four-byte id and a
// four-byte distance plane and a merged hull per row they took 39 + 9 us and
// 217 us.  With 200 000 clustered seeds 35 and 110 us against 45 + 10 and
// 249 us; the rows of 512 batch images 0.68 ms against 2.8 ms.
#include "context.cuh"
#include "exact_pass.cuh"

#include <atomic>
#include <type_traits>

namespace idl {
namespace {

__global__ void __launch_bounds__(64)
k_column_off(const uint32_t* __restrict__ pos, SeedRanks ranks, XImg m, int pitch, int16_t* __restrict__ off,
             uint4* __restrict__ bands)
{
    const int c = (blockIdx.x * 64 + threadIdx.x) * 2;
    if (c < m.Wp) x_column_pair(pos, ranks, m, c, blockIdx.y, pitch, off, bands);
}

__global__ void __launch_bounds__(64)
k_bx_column_off(const uint32_t* __restrict__ pos, SeedRanks ranks, const XImg* __restrict__ xi,
                const int32_t* __restrict__ pair_img, int n_pairs, int pitch, int16_t* __restrict__ off,
                uint4* __restrict__ bands)
{
    const int g = blockIdx.x * 64 + threadIdx.x;
    if (g >= n_pairs) return;
    const XImg m = xi[pair_img[g]];
    if ((int)blockIdx.y < x_bands(m)) x_column_pair(pos, ranks, m, (g - m.pair_off) * 2, blockIdx.y, pitch, off, bands);
}

// Image of each column pair and row of the batch; a block per image.
__global__ void k_bx_tables(const XImg* __restrict__ xi, int32_t* __restrict__ pair_img, int32_t* __restrict__ row_img)
{
    const XImg& m = xi[blockIdx.x];
    for (int i = threadIdx.x; i < (m.Wp + 1) / 2; i += blockDim.x) pair_img[m.pair_off + i] = blockIdx.x;
    for (int i = threadIdx.x; i < m.Hp; i += blockDim.x) row_img[m.row_off + i] = blockIdx.x;
}

template <int T, bool LABELS>
__global__ void __launch_bounds__(T)
k_row_win(const int16_t* __restrict__ off, XImg m, int pitch, SeedBands seeds, int32_t* __restrict__ lab,
          int list_bytes)
{
    const int y = blockIdx.x;
    x_row<T, LABELS>(off + (size_t)y * pitch, y, m, seeds, lab + (size_t)y * pitch, list_bytes);
}

template <int T>
__global__ void __launch_bounds__(T)
k_bx_row_win(const int16_t* __restrict__ off, const XImg* __restrict__ xi, const int32_t* __restrict__ row_img,
             int pitch, SeedBands seeds, int32_t* __restrict__ lab, int list_bytes)
{
    const XImg m = xi[row_img[blockIdx.x]];
    const int y = m.oy + (int)blockIdx.x - m.row_off;
    const size_t o = (size_t)y * pitch + m.ox;
    x_row<T, false>(off + o, y, m, seeds, lab + o, list_bytes);
}

template <class K, class... A>
void launch_rows(Context& C, K kernel, std::atomic<uint64_t>& opted, unsigned rows, int threads, size_t smem, A... args)
{
    // the shared-memory opt-in is per device
    const uint64_t bit = 1ull << (C.device & 63);
    if (!(opted.load(std::memory_order_acquire) & bit)) {
        IDL_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 256));
        opted.fetch_or(bit, std::memory_order_acq_rel);
    }
    kernel<<<rows, threads, smem, C.stream>>>(args...);
    IDL_LAUNCH();
}

// One instantiation per row width class (row_pass_threads): which(threads)
// names the kernel.
template <class W, class... A>
void rows_for_width(Context& C, int width, unsigned rows, std::atomic<uint64_t>* opted, W&& which, A... args)
{
    const int threads = row_pass_threads(width, rows);
    const size_t smem = row_pass_smem(width);
    auto go = [&](auto tag, int slot) {
        launch_rows(C, which(tag), opted[slot], rows, threads, smem, args..., row_list_bytes(width));
    };
    if (threads == 32) go(std::integral_constant<int, 32>{}, 0);
    else if (threads == 64) go(std::integral_constant<int, 64>{}, 1);
    else if (threads == 128) go(std::integral_constant<int, 128>{}, 2);
    else if (threads == 256) go(std::integral_constant<int, 256>{}, 3);
    else go(std::integral_constant<int, 1024>{}, 4);
}

}  // namespace

XImg whole_canvas(const Canvas& cv, int64_t n, int P)
{
    XImg m{};
    m.Wp = cv.Wd;
    m.Hp = cv.Hd;
    m.s1 = (int)n;
    m.P = P;
    return m;
}

void propagate_exact(Context& C, const Canvas& cv, const uint32_t* pos, int64_t n, int P, const int32_t* label)
{
    const size_t plane = (size_t)cv.pitch * cv.Hd * 4;
    C.lab[0].ensure(plane);
    C.lab[1].ensure(plane);
    const XImg m = whole_canvas(cv, n, P);
    C.exact_bands.ensure((size_t)x_bands(m) * cv.Wd * sizeof(uint4));
    int16_t* off = C.lab[1].as<int16_t>();
    uint4* bands = C.exact_bands.as<uint4>();
    const SeedRanks ranks{C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), label};
    const SeedBands seeds{bands, label};
    k_column_off<<<dim3((unsigned)ceil_div(cv.Wd, 128), (unsigned)x_bands(m)), 64, 0, C.stream>>>(pos, ranks, m, cv.pitch,
                                                                                               off, bands);
    IDL_LAUNCH();
    static std::atomic<uint64_t> opted[2][5];
    const int16_t* o = off;
    if (label)
        rows_for_width(C, cv.Wd, (unsigned)cv.Hd, opted[1], [](auto T) { return k_row_win<T(), true>; }, o, m, cv.pitch,
                       seeds, C.lab[0].as<int32_t>());
    else
        rows_for_width(C, cv.Wd, (unsigned)cv.Hd, opted[0], [](auto T) { return k_row_win<T(), false>; }, o, m,
                       cv.pitch, seeds, C.lab[0].as<int32_t>());
    if (C.prof.enabled) {
        C.prof.passes = 0;
        C.prof.rounds = 2;
        C.prof.tiles = 0;
        C.prof.prop_bytes = (double)cv.Wd * cv.Hd * 8.0;   // column offsets out and in, labels out
        C.prof.tile_w = C.prof.tile_h = 0;
        C.prof.steps_per_round = 0;
    }
}

void exact_images(Context& C, int pitch, const uint32_t* pos, const XImg* xi, int n_images, int32_t* pair_img,
                  int n_pairs, int32_t* row_img, int n_rows, int max_wp, int max_hp, int64_t band_entries)
{
    k_bx_tables<<<(unsigned)n_images, 256, 0, C.stream>>>(xi, pair_img, row_img);
    IDL_LAUNCH();
    int16_t* off = C.lab[1].as<int16_t>();
    C.exact_bands.ensure((size_t)band_entries * sizeof(uint4));
    uint4* bands = C.exact_bands.as<uint4>();
    const SeedRanks ranks{C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), nullptr};
    const SeedBands seeds{bands, nullptr};
    k_bx_column_off<<<dim3((unsigned)ceil_div(n_pairs, 64), (unsigned)ceil_div(max_hp, BAND)), 64, 0, C.stream>>>(
        pos, ranks, xi, pair_img, n_pairs, pitch, off, bands);
    IDL_LAUNCH();
    static std::atomic<uint64_t> opted[5];
    rows_for_width(C, max_wp, (unsigned)n_rows, opted, [](auto T) { return k_bx_row_win<T()>; }, (const int16_t*)off, xi,
                   (const int32_t*)row_img, pitch, seeds, C.lab[0].as<int32_t>());
}

}  // namespace idl
