// Seed validation and (x, y) ordering on the device, plus the exclusive scan
// the rest of the library shares.
//
// The reference sorts seeds on the host with std::sort after a Python-object
// loop (src/cuda/bindings/binding_helpers.hpp:23-46).  Seeds are distinct
// pixels, so their (x asc, y asc) order is the order of their pixels in a
// column-major walk of the canvas: set one bit per seed in a column-major
// occupancy bitmap (a repeat hit is a duplicate), prefix-popcount the bitmap,
// and each seed's rank is the number of set bits before its own.  O(n + W*H/32)
// work, no comparison sort, and the duplicate check falls out of the atomicOr.
#include "context.cuh"

#include <vector>

namespace idl {

// ---------------------------------------------------------------------------
// exclusive scan (int32, or of the popcounts of 32-bit words): per-block sums,
// scanned by the block that finishes last, then the blocks' own scans on top.
// Two launches, one for up to SCAN_TILE items: on a small image the launches
// of a scan level by level cost more than the scan.
// ---------------------------------------------------------------------------
namespace {

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <bool POPC>
__device__ __forceinline__ int32_t scan_item(const int32_t* __restrict__ in, int64_t j, int64_t n)
{
    if (j >= n) return 0;
    return POPC ? __popc((uint32_t)in[j]) : in[j];
}

// Exclusive prefix of v over the block's threads; *total: their sum.
__device__ __forceinline__ int32_t block_prefix(int32_t v, int32_t* total)
{
    __shared__ int32_t warp_sum[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    int32_t before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < SCAN_THREADS / 32; ++k) {
        const int32_t w = warp_sum[k];
        before += k < warp ? w : 0;
        all += w;
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

template <bool POPC>
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_sums(const int32_t* __restrict__ in, int64_t n, int32_t* __restrict__ sums, int32_t* __restrict__ total,
            int32_t* __restrict__ done)
{
    __shared__ bool last;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    int32_t v = 0, all;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) v += scan_item<POPC>(in, base + i * SCAN_THREADS + threadIdx.x, n);
    block_prefix(v, &all);
    if (threadIdx.x == 0) {
        sums[blockIdx.x] = all;
        __threadfence();
        last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int32_t carry = 0;
    for (unsigned b0 = 0; b0 < gridDim.x; b0 += SCAN_THREADS) {
        const unsigned b = b0 + threadIdx.x;
        const int32_t s = b < gridDim.x ? __ldcg(&sums[b]) : 0;
        const int32_t before = block_prefix(s, &all);
        if (b < gridDim.x) sums[b] = carry + before;
        carry += all;
    }
    if (threadIdx.x == 0) {
        *total = carry;
        *done = 0;   // for the next scan on this context
    }
}

template <bool POPC>
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_write(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t n, const int32_t* __restrict__ sums)
{
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
    int32_t v[SCAN_ITEMS];
    int32_t run = 0, all;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        v[i] = run;
        run += scan_item<POPC>(in, base + i, n);
    }
    const int32_t before = (sums ? sums[blockIdx.x] : 0) + block_prefix(run, &all);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i)
        if (base + i < n) out[base + i] = before + v[i];
    if (!sums && threadIdx.x == 0) out[n] = all;
}

template <bool POPC>
void scan(Context& C, const int32_t* in, int32_t* out, int64_t n)
{
    const int64_t nb = std::max<int64_t>(1, (n + SCAN_TILE - 1) / SCAN_TILE);
    int32_t* sums = nullptr;
    if (nb > 1) {
        C.scan_a.ensure((size_t)nb * sizeof(int32_t));
        sums = C.scan_a.as<int32_t>();
        k_scan_sums<POPC><<<(unsigned)nb, SCAN_THREADS, 0, C.stream>>>(in, n, sums, out + n, &C.sc()->scan_done);
        IDL_LAUNCH();
    }
    k_scan_write<POPC><<<(unsigned)nb, SCAN_THREADS, 0, C.stream>>>(in, out, n, sums);
    IDL_LAUNCH();
}

}  // namespace

void exclusive_scan(Context& C, const int32_t* in, int32_t* out, int64_t n) { scan<false>(C, in, out, n); }

void exclusive_popc_scan(Context& C, const uint32_t* words, int32_t* out, int64_t n)
{
    scan<true>(C, reinterpret_cast<const int32_t*>(words), out, n);
}

// ---------------------------------------------------------------------------
// seeds
// ---------------------------------------------------------------------------
namespace {

__global__ void k_seed_mark(const int32_t* __restrict__ xy, int64_t n, int W, int H,
                            uint32_t* __restrict__ bitmap, Scalars* __restrict__ sc)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int x = xy[2 * i], y = xy[2 * i + 1];
    if (x < 0 || x >= W || y < 0 || y >= H) {
        atomicOr(&sc->err_oob, 1);
        return;
    }
    const int64_t bit = (int64_t)x * H + y;
    const uint32_t m = 1u << (bit & 31);
    const uint32_t old = atomicOr(&bitmap[bit >> 5], m);
    if (old & m) atomicOr(&sc->err_dup, 1);
}

__global__ void k_seed_rank(const int32_t* __restrict__ xy, int64_t n, int W, int H, int P,
                            const uint32_t* __restrict__ bitmap, const int32_t* __restrict__ word_rank,
                            int32_t* __restrict__ xs, int32_t* __restrict__ ys, uint32_t* __restrict__ pos)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int x = xy[2 * i], y = xy[2 * i + 1];
    if (x < 0 || x >= W || y < 0 || y >= H) return;
    const int64_t bit = (int64_t)x * H + y;
    const uint32_t below = bitmap[bit >> 5] & ((1u << (bit & 31)) - 1u);
    const int32_t r = word_rank[bit >> 5] + __popc(below);
    xs[r] = x;
    ys[r] = y;
    pos[r] = pack_pos(x + P, y + P);
}

__global__ void k_mark_xy(const int32_t* __restrict__ xs, const int32_t* __restrict__ ys, int64_t n, int H,
                          uint32_t* __restrict__ bitmap)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t bit = (int64_t)xs[i] * H + ys[i];
    atomicOr(&bitmap[bit >> 5], 1u << (bit & 31));
}

__global__ void k_rank_xy(const int32_t* __restrict__ xs, const int32_t* __restrict__ ys, int64_t n, int H,
                          const uint32_t* __restrict__ bitmap, const int32_t* __restrict__ word_rank, int off,
                          int32_t* __restrict__ rank, int32_t* __restrict__ inv, int32_t* __restrict__ xs_sorted,
                          int32_t* __restrict__ ys_sorted)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t bit = (int64_t)xs[i] * H + ys[i];
    const uint32_t below = bitmap[bit >> 5] & ((1u << (bit & 31)) - 1u);
    const int32_t r = word_rank[bit >> 5] + __popc(below);
    rank[i] = r;
    inv[r] = (int32_t)i;
    xs_sorted[r] = xs[i] + off;
    ys_sorted[r] = ys[i] + off;
}

}  // namespace

void rank_seeds_device(Context& C, int W, int H, const int32_t* xs, const int32_t* ys, int64_t n, int off,
                       int32_t* rank, int32_t* inv, int32_t* xs_sorted, int32_t* ys_sorted)
{
    if (n <= 0) return;
    const int64_t nwords = ((int64_t)W * H + 31) / 32;
    C.bitmap.ensure(size_t(nwords) * 4);
    C.scan_c.ensure(size_t(nwords + 1) * 4);
    // with the bits, the scan's counter, so that no earlier state of it matters
    ClearList zero;
    zero.add(C.bitmap.ptr, size_t(nwords) * 4, 0);
    zero.add(reinterpret_cast<char*>(C.sc()) + SCAN_UNIT, 16, 0);
    clear_buffers(C, zero);
    const unsigned gs = (unsigned)((n + 255) / 256);
    k_mark_xy<<<gs, 256, 0, C.stream>>>(xs, ys, n, H, C.bitmap.as<uint32_t>());
    IDL_LAUNCH();
    exclusive_popc_scan(C, C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), nwords);
    k_rank_xy<<<gs, 256, 0, C.stream>>>(xs, ys, n, H, C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), off, rank,
                                        inv, xs_sorted, ys_sorted);
    IDL_LAUNCH();
}

void sort_seeds_device(Context& C, int W, int H, int64_t n, int P)
{
    const int64_t bits = (int64_t)W * H;
    const int64_t nwords = (bits + 31) / 32;
    C.bitmap.ensure(size_t(nwords) * 4);
    C.scan_c.ensure(size_t(nwords + 1) * 4);
    C.xs.ensure(size_t(n) * 4);
    C.ys.ensure(size_t(n) * 4);
    C.pos.ensure(size_t(n) * 4);

    if (!C.precleared) {
        IDL_CUDA(cudaMemsetAsync(C.bitmap.ptr, 0, size_t(nwords) * 4, C.stream));
        IDL_CUDA(cudaMemsetAsync(&C.sc()->err_oob, 0, 3 * sizeof(int32_t), C.stream));
    }
    const unsigned gs = (unsigned)((n + 255) / 256);
    k_seed_mark<<<gs, 256, 0, C.stream>>>(C.seeds_in.as<int32_t>(), n, W, H, C.bitmap.as<uint32_t>(), C.sc());
    IDL_LAUNCH();
    C.fetch_scalars_begin();
    exclusive_popc_scan(C, C.bitmap.as<uint32_t>(), C.scan_c.as<int32_t>(), nwords);
    k_seed_rank<<<gs, 256, 0, C.stream>>>(C.seeds_in.as<int32_t>(), n, W, H, P, C.bitmap.as<uint32_t>(),
                                          C.scan_c.as<int32_t>(), C.xs.as<int32_t>(), C.ys.as<int32_t>(),
                                          C.pos.as<uint32_t>());
    IDL_LAUNCH();
    // the flags are waited for with the ranking already queued behind them (it
    // stays in bounds on seeds that are about to be refused)
    C.fetch_scalars_end();
    if (C.host_sc->err_oob) invalid("seed coordinate out of bounds");
    if (C.host_sc->err_dup) invalid("duplicate seed positions are not allowed");
}

}  // namespace idl
