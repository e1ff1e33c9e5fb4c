// C ABI: context management and the batch entry points (Voronoi().compute,
// triangulate(), GridTriangulation.compute*), plus the output composition
// kernels.  The orchestration follows cuda_compute_triangulation
// (src/cuda/triangulation.cu:143-365) stage for stage, with every
// intermediate kept on the device and no host loops over pixels.
#include "context.cuh"

#include <algorithm>
#include <atomic>
#include <string>

namespace idl {

namespace {
thread_local std::string g_last_error;
std::atomic<long long> g_launches{0};
std::atomic<long long> g_allocs{0};
}

void set_last_error(const char* msg) { g_last_error = msg ? msg : ""; }
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void count_alloc() { g_allocs.fetch_add(1, std::memory_order_relaxed); }

size_t Context::workspace_bytes() const
{
    size_t s = 0;
    const_cast<Context*>(this)->each_buf([&](DevBuf& b) { s += b.bytes; });
    return s;
}

void Context::fetch_scalars()
{
    IDL_CUDA(cudaMemcpyAsync(host_sc, scalars.ptr, sizeof(Scalars), cudaMemcpyDeviceToHost, stream));
    IDL_CUDA(cudaStreamSynchronize(stream));
}

void Context::fetch_scalars_begin()
{
    IDL_CUDA(cudaMemcpyAsync(host_sc, scalars.ptr, sizeof(Scalars), cudaMemcpyDeviceToHost, stream));
    if (host_sc_borrowed) return;   // a pageable mirror: the copy is done when the call returns
    if (!fetched) IDL_CUDA(cudaEventCreateWithFlags(&fetched, cudaEventDisableTiming));
    IDL_CUDA(cudaEventRecord(fetched, stream));
}

void Context::fetch_scalars_end()
{
    if (host_sc_borrowed) IDL_CUDA(cudaStreamSynchronize(stream));
    else IDL_CUDA(cudaEventSynchronize(fetched));
}

Context::~Context()
{
    if (fetched) cudaEventDestroy(fetched);
    bool ordered = false;
    each_buf([&](DevBuf& b) { ordered |= b.async; });
    if (ordered) cudaDeviceSynchronize();   // stream-ordered buffers may still be in use
    each_buf([](DevBuf& b) { b.release(); });
    if (host_sc && !host_sc_borrowed) cudaFreeHost(host_sc);
    for (auto& e : timing.ev)
        if (e) cudaEventDestroy(e);
}

void ensure_scalars(Context& C)
{
    if (!C.scalars.ptr) {
        C.scalars.ensure(sizeof(Scalars));
        IDL_CUDA(cudaMemsetAsync(C.scalars.ptr, 0, sizeof(Scalars), C.stream));
    }
    if (!C.host_sc) {
        count_alloc();
        IDL_CUDA(cudaMallocHost(reinterpret_cast<void**>(&C.host_sc), sizeof(Scalars)));
    }
}

namespace {

__global__ void __launch_bounds__(256) k_clear(ClearList l)
{
    const long long step = (long long)gridDim.x * blockDim.x;
    for (int k = 0; k < l.count; ++k) {
        const uint32_t v = l.word[k];
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < l.n[k]; i += step)
            l.p[k][i] = make_uint4(v, v, v, v);
    }
}

}  // namespace

void clear_buffers(Context& C, const ClearList& l)
{
    long long units = 1;
    for (int k = 0; k < l.count; ++k) units = std::max(units, l.n[k]);
    const unsigned blocks = (unsigned)std::min<long long>((units + 255) / 256, C.num_sms * 16);
    k_clear<<<blocks, 256, 0, C.stream>>>(l);
    IDL_LAUNCH();
}

void clear_for_run(Context& C, const Canvas& cv, int W, int H, int64_t n, bool suspects, int64_t cap, int64_t n_tri)
{
    C.owner = nullptr;   // the counters are the run's from here on
    ClearList l;
    const size_t bitmap = ((size_t)W * H + 31) / 32 * 4;
    C.bitmap.ensure(bitmap);
    l.add(C.scalars.ptr, sizeof(Scalars), 0);
    l.add(C.bitmap.ptr, bitmap, 0);
    if (suspects) {
        const size_t bits = resolve_reserve(C, cv);
        l.add(C.sus_bits.ptr, bits, 0);
    }
    if (cap > 0) {
        detect_reserve(C, n, cap);
        l.add(C.hkeys.ptr, (size_t)cap * 16, 0xFFFFFFFFu);
        l.add(C.cnt.ptr, (size_t)(n + 1) * 2 * 4, 0);
        const size_t head = raster_reserve(C, W, H, n_tri);
        l.add(C.rbig.ptr, head, 0);
    }
    clear_buffers(C, l);
    C.precleared = true;
}

namespace {

// Ends a run's use of cleared buffers, however the run ends.
struct Precleared {
    Context& C;
    ~Precleared() { C.precleared = false; }
};

// ---- output composition ------------------------------------------------

// (a, b, c) of each (x, y, a, b, c) triangle row.
__global__ void k_tri_vertices(const int32_t* __restrict__ tris, int64_t n, int32_t* __restrict__ verts)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * 3) return;
    const int64_t t = i / 3;
    verts[i] = tris[t * 5 + 2 + (i - t * 3)];
}

// GridTriangulation at P == 0 with the caller's grid: channels 0 and 1 are the
// caller's (triangulation.cu:406-411).
__global__ void k_compose3_from_grid(const int32_t* __restrict__ vgrid, int W, int H,
                                     const int32_t* __restrict__ tgrid, int32_t* __restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const size_t i = (size_t)y * W + x;
    out[i * 3] = vgrid[i * 2];
    out[i * 3 + 1] = vgrid[i * 2 + 1];
    out[i * 3 + 2] = tgrid[i];
}

// (H, W, 2) seed id + squared distance of a label plane (Voronoi().compute,
// and compute_debug's padded grid).  pos holds coordinates of the same canvas.
__global__ void k_compose2(const int32_t* __restrict__ lab, int pitch, int W, int H,
                           const uint32_t* __restrict__ pos, int32_t* __restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const int32_t l = lab[(size_t)y * pitch + x];
    const size_t i = (size_t)y * W + x;
    out[i * 2] = l;
    out[i * 2 + 1] = l >= 0 ? dist2(x, y, __ldg(&pos[l])) : -1;
}

// Label plane from a caller's (H, W, 2) grid, with the ids checked against
// the seed count (the reference indexes its seed arrays with them unchecked).
__global__ void k_labels_from_grid(const int32_t* __restrict__ vgrid, int W, int H, int pitch, int64_t n,
                                   int32_t* __restrict__ lab, Scalars* __restrict__ sc)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const int32_t l = vgrid[((size_t)y * W + x) * 2];
    if (l < -1 || l >= n) atomicOr(&sc->err_label, 1);
    lab[(size_t)y * pitch + x] = (l < -1 || l >= n) ? UNDEF : l;
}

int resolve_padding(int p)
{
    // binding_helpers.hpp:49-53: only the sentinel means "default".  Other
    // negatives are clamped to 0, as the NumPy reference does
    // (reference/triangulation.py:78); the reference CUDA path has no
    // defined behaviour for them.
    if (p == IDL_AUTO_BORDER_PADDING) return IDL_DEFAULT_BORDER_PADDING;
    return p < 0 ? 0 : p;
}

void check_mode(int mode)
{
    if (mode != IDL_MODE_REFERENCE && mode != IDL_MODE_NUMPY && mode != IDL_MODE_EXACT)
        invalid("mode must be one of IDL_MODE_REFERENCE, IDL_MODE_NUMPY, IDL_MODE_EXACT");
}

Canvas make_canvas(int Wd, int Hd)
{
    if (Wd > MAX_CANVAS_SIDE || Hd > MAX_CANVAS_SIDE)
        invalid("canvas side (including border padding) must not exceed " + std::to_string(MAX_CANVAS_SIDE));
    Canvas cv;
    cv.Wd = Wd;
    cv.Hd = Hd;
    cv.pitch = (Wd + 31) / 32 * 32;
    return cv;
}

void check_seed_count(int64_t n)
{
    if (n <= 0) invalid("seeds must not be empty");
    if (n > MAX_SEEDS) invalid("at most " + std::to_string(MAX_SEEDS) + " seeds are supported");
}

struct StageTimer {
    Context& C;
    bool on;
    StageTimer(Context& c, bool enable) : C(c), on(enable)
    {
        if (!on) return;
        for (auto& e : C.timing.ev)
            if (!e) IDL_CUDA(cudaEventCreate(&e));
    }
    void mark(int i)
    {
        if (on) IDL_CUDA(cudaEventRecord(C.timing.ev[i], C.stream));
    }
    float ms(int a, int b)
    {
        float t = 0.f;
        if (on) IDL_CUDA(cudaEventElapsedTime(&t, C.timing.ev[a], C.timing.ev[b]));
        return t;
    }
};

// Stage (a) by running the passes, from the sorted seeds of C.pos.
int64_t run_passes(Context& C, int mode, const Canvas& cv, int64_t n)
{
    init_labels(C, cv, C.pos.as<uint32_t>(), n);
    return propagate(C, mode, cv, C.pos.as<uint32_t>(), n);
}

// Stage (a) from scratch into C.lab[0].  Returns true if the labels come from
// resolve_exact: the caller has to look at resolved() once the scalars have been
// read back.  Otherwise *passes (may be nullptr) takes the pass count.
bool start_labels(Context& C, int mode, const Canvas& cv, int64_t n, int P, int64_t* passes = nullptr)
{
    if (mode == IDL_MODE_REFERENCE && C.direct()) {
        C.prof.pass_ns.clear();
        C.prof.pass_tiles.clear();
        propagate_exact(C, cv, C.pos.as<uint32_t>(), n, P);
        resolve_exact(C, cv, C.pos.as<uint32_t>(), n);
        return true;
    }
    int64_t p = 0;
    if (mode == IDL_MODE_EXACT) propagate_exact(C, cv, C.pos.as<uint32_t>(), n, P);
    else p = run_passes(C, mode, cv, n);
    if (passes) *passes = p;
    return false;
}

// The pass count of labels that stand, after resolve_arrivals and a read-back of
// the scalars.  Where those do not determine it, the passes are run after all;
// they reach the same labels, and a profile keeps what it has recorded.
int64_t count_passes(Context& C, int mode, const Canvas& cv, int64_t n)
{
    int64_t p = resolved_passes(*C.host_sc);
    if (p < 0) {
        const Profile kept = C.prof;
        C.prof.enabled = false;
        p = run_passes(C, mode, cv, n);
        C.prof = kept;
    }
    return p;
}

// Run stages (a) (b) (d) with seeds already in C.seeds_in.  Leaves labels in
// C.lab[0], triangles in C.tris, the composed (H, W, 3) grid in d_out; deliver()
// queues the copies the caller wants of them.  Returns the triangle count, with
// the stream's work done.
template <class F>
int64_t run_triangulate(Context& C, int W, int H, int64_t n, const int32_t* vgrid, int P, int mode, float* timings,
                        int32_t* d_out, F&& deliver)
{
    const Canvas cv = make_canvas(W + 2 * P, H + 2 * P);
    C.prof.valid = false;
    for (bool& r : C.prof.recorded) r = false;
    C.prof.rounds = C.prof.tiles = C.prof.passes = 0;
    C.prof.prop_bytes = 0;
    // the usual bounds on the hash table and the triangle count (under 2n)
    int64_t cap = detect_capacity(C, n);
    const int64_t bound = C.selftest.bound(IDL_LIMIT_TRIANGLES, 2 * n + 64);
    const bool from_grid = vgrid && P == 0;
    C.mark(PM_START);
    const Precleared guard{C};
    clear_for_run(C, cv, W, H, n, !from_grid && mode == IDL_MODE_REFERENCE && C.direct(), cap, bound);
    sort_seeds_device(C, W, H, n, P);
    C.mark(PM_SEEDS);

    bool resolved = false;
    if (!from_grid) {
        resolved = start_labels(C, mode, cv, n, P);
    } else {
        const size_t gbytes = (size_t)W * H * 2 * sizeof(int32_t);
        C.vgrid.ensure(gbytes);
        IDL_CUDA(cudaMemcpyAsync(C.vgrid.ptr, vgrid, gbytes, cudaMemcpyHostToDevice, C.stream));
        C.lab[0].ensure((size_t)cv.pitch * cv.Hd * 4);
        IDL_CUDA(cudaMemsetAsync(&C.sc()->err_label, 0, sizeof(int32_t), C.stream));
        dim3 g(ceil_div(W, 256), H);
        k_labels_from_grid<<<g, 256, 0, C.stream>>>(C.vgrid.as<int32_t>(), W, H, cv.pitch, n, C.lab[0].as<int32_t>(),
                                                   C.sc());
        IDL_LAUNCH();
        C.fetch_scalars();
        if (C.host_sc->err_label) invalid("voronoi_grid seed ids must lie in [-1, number of seeds)");
    }
    C.mark(PM_PROPAGATE);

    StageTimer T(C, timings != nullptr);
    const int32_t *xs = C.xs.as<int32_t>(), *ys = C.ys.as<int32_t>();
    auto detect = [&](int64_t cap) {
        T.mark(0);
        // detect_ms covers the fused detect + hash insert kernel, dedup_ms the
        // enumeration and canonical ranking (the reference's thrust sort/unique)
        detect_launch(C, cv, C.lab[0].as<int32_t>(), C.pos.as<uint32_t>(), n, P, cap, T.on ? C.timing.ev[1] : nullptr);
        T.mark(2);
        C.mark(PM_DEDUP);
    };
    auto assign = [&](int64_t n_tri) {
        T.mark(3);
        if (from_grid) {   // channels 0 and 1 are the caller's
            C.tgrid.ensure((size_t)W * H * sizeof(int32_t));
            assign_pixels(C, W, H, xs, ys, C.tgrid.as<int32_t>(), n_tri, true);
            C.mark(PM_ASSIGN);
            k_compose3_from_grid<<<dim3(ceil_div(W, 256), H), 256, 0, C.stream>>>(C.vgrid.as<int32_t>(), W, H,
                                                                                 C.tgrid.as<int32_t>(), d_out);
            IDL_LAUNCH();
        } else {
            assign_and_compose(C, W, H, xs, ys, n_tri, C.lab[0].as<int32_t>() + (size_t)P * cv.pitch + P, cv.pitch,
                               d_out);
            C.mark(PM_ASSIGN);
        }
        C.mark(PM_COMPOSE);
        T.mark(4);
        if (resolved && C.prof.enabled) resolve_arrivals(C, cv, C.pos.as<uint32_t>());
        deliver(cv);
        C.fetch_scalars();
    };
    // Everything after the seeds' check goes out before anything is read back; one
    // wait at the end tells whether the bounds held and whether the exact diagram decided the
    // labels.  What failed is run again, each time with room for what is known
    // by then (more triangles than `bound`, as a caller's grid can hold, are not
    // drawn in vain).
    detect(cap);
    assign(bound);
    C.precleared = false;
    if (resolved && !idl::resolved(C)) {
        resolved = false;
        run_passes(C, mode, cv, n);
        C.mark(PM_PROPAGATE);
        detect(cap);
        assign(bound);
    }
    for (int attempt = 0; !detect_done(C, cap); ++attempt) {
        if (attempt >= 6) throw Error(IDL_ERR_INTERNAL, "triangle hash table overflow");
        cap *= 4;
        detect(cap);
        assign(bound);
    }
    if (C.host_sc->n_triangles > bound) assign(C.host_sc->n_triangles);
    const int64_t nt = C.host_sc->n_triangles;
    if (resolved && C.prof.enabled) C.prof.passes = count_passes(C, mode, cv, n);
    if (timings) {
        timings[IDL_T_DETECT_MS] = T.ms(0, 1);
        timings[IDL_T_DEDUP_MS] = T.ms(1, 2);
        timings[IDL_T_ASSIGN_MS] = T.ms(3, 4);
    }
    C.last_n_tri = nt;
    C.have_result = true;
    C.prof.canvas_px = (int64_t)cv.Wd * cv.Hd;
    C.prof.image_px = (int64_t)W * H;
    C.prof.n_triangles = nt;
    C.prof.valid = C.prof.enabled;
    return nt;
}

void upload_seeds(Context& C, const int32_t* xy, int64_t n, cudaMemcpyKind kind)
{
    C.seeds_in.ensure((size_t)n * 2 * sizeof(int32_t));
    IDL_CUDA(cudaMemcpyAsync(C.seeds_in.ptr, xy, (size_t)n * 2 * sizeof(int32_t), kind, C.stream));
}

void check_dims(int W, int H, int64_t n)
{
    if (W <= 0 || H <= 0) {
        if (n <= 0) invalid("seeds must not be empty");
        invalid("seed coordinate out of bounds");
    }
}

}  // namespace
}  // namespace idl

using namespace idl;


extern "C" {

const char* idl_last_error(void) { return g_last_error.c_str(); }

int idl_version(void) { return 100; }

long long idl_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

long long idl_alloc_count(void) { return g_allocs.load(std::memory_order_relaxed); }

int idl_selftest_grid_barrier(idl_context* ctx, int missing_arrivals, unsigned int spin_limit)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    DeviceGuard g(ctx->device);
    grid_barrier_selftest(*ctx, missing_arrivals, spin_limit);
    IDL_API_END
}

int idl_selftest_limit(idl_context* ctx, int which, int64_t limit)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (which < 0 || which >= IDL_LIMIT_COUNT) invalid("no such limit");
    if (limit < 0) invalid("limit must not be negative");
    ctx->selftest.limit[which] = limit;
    IDL_API_END
}

int idl_selftest_counts(idl_context* ctx, int64_t* out, int n)
{
    IDL_API_BEGIN
    if (!ctx || !out) invalid("arguments must not be NULL");
    for (int i = 0; i < n && i < IDL_COUNTED; ++i) out[i] = ctx->selftest.count[i];
    IDL_API_END
}

int idl_context_create(int device, idl_context** out)
{
    IDL_API_BEGIN
    if (!out) invalid("out must not be NULL");
    *out = nullptr;
    int dev = device;
    if (dev < 0) IDL_CUDA(cudaGetDevice(&dev));
    DeviceGuard g(dev);
    auto* c = new idl_context();
    c->device = dev;
    try {
        IDL_CUDA(cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, dev));
        ensure_scalars(*c);
    } catch (...) {
        delete c;
        throw;
    }
    *out = c;
    IDL_API_END
}

int idl_context_destroy(idl_context* ctx)
{
    IDL_API_BEGIN
    if (!ctx) return IDL_OK;
    DeviceGuard g(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    delete ctx;
    IDL_API_END
}

int idl_context_set_stream(idl_context* ctx, void* stream)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    const cudaStream_t next = static_cast<cudaStream_t>(stream);
    // Workspace growth is freed in the order of the context's stream: finish
    // the old stream's work before later frees are ordered on the new one.
    if (next != ctx->stream) {
        DeviceGuard g(ctx->device);
        IDL_CUDA(cudaStreamSynchronize(ctx->stream));
    }
    ctx->stream = next;
    IDL_API_END
}

int idl_context_set_schedule(idl_context* ctx, int dense_rounds)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    ctx->dense_rounds = dense_rounds;
    IDL_API_END
}

int idl_context_set_tile(idl_context* ctx, int shape, int* n_shapes_out)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (n_shapes_out) *n_shapes_out = key_tile_shapes();
    if (shape < 0 || shape >= key_tile_shapes()) invalid("tile shape index out of range");
    ctx->key_tile = shape;
    IDL_API_END
}

int idl_context_synchronize(idl_context* ctx)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    DeviceGuard g(ctx->device);
    IDL_CUDA(cudaStreamSynchronize(ctx->stream));
    IDL_API_END
}

int idl_context_workspace_bytes(idl_context* ctx, int64_t* bytes_out)
{
    IDL_API_BEGIN
    if (!ctx || !bytes_out) invalid("arguments must not be NULL");
    *bytes_out = (int64_t)ctx->workspace_bytes();
    IDL_API_END
}

int idl_context_set_profiling(idl_context* ctx, int enable)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    ctx->prof.enabled = enable != 0;
    ctx->prof.valid = false;
    IDL_API_END
}

int idl_context_pass_trace(idl_context* ctx, int64_t* ns_out, int32_t* tiles_out, int32_t* steps_out, int capacity,
                           int* n_out)
{
    IDL_API_BEGIN
    if (!ctx || !n_out) invalid("arguments must not be NULL");
    const Profile& P = ctx->prof;
    *n_out = (int)P.pass_ns.size();
    for (int i = 0; i < capacity && i < (int)P.pass_ns.size(); ++i) {
        if (ns_out) ns_out[i] = P.pass_ns[i];
        if (tiles_out) tiles_out[i] = P.pass_tiles[i];
        if (steps_out) steps_out[i] = i < (int)P.pass_steps.size() ? P.pass_steps[i] : 1;
    }
    IDL_API_END
}

int idl_context_set_tail_rounds(idl_context* ctx, int max_list)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (max_list < 0) invalid("max_list must not be negative");
    ctx->tail_rounds_below = max_list;
    IDL_API_END
}

int idl_context_last_profile(idl_context* ctx, double* out, int n)
{
    IDL_API_BEGIN
    if (!ctx || !out) invalid("arguments must not be NULL");
    if (!ctx->prof.valid) throw Error(IDL_ERR_STATE, "no profiled run on this context");
    DeviceGuard g(ctx->device);
    Profile& P = ctx->prof;
    double v[IDL_PROF_COUNT] = {};
    for (int m = PM_SEEDS; m < PM_COUNT; ++m) {
        int prev = m - 1;
        while (prev > PM_START && !P.recorded[prev]) --prev;
        if (P.recorded[m] && P.recorded[prev]) {
            IDL_CUDA(cudaEventSynchronize(P.ev[m]));
            float ms = 0.f;
            IDL_CUDA(cudaEventElapsedTime(&ms, P.ev[prev], P.ev[m]));
            v[m - 1] = ms;
        }
    }
    v[IDL_PROF_ROUNDS] = (double)P.rounds;
    v[IDL_PROF_TILES] = (double)P.tiles;
    v[IDL_PROF_PASSES] = (double)P.passes;
    v[IDL_PROF_TILE_W] = P.tile_w;
    v[IDL_PROF_TILE_H] = P.tile_h;
    v[IDL_PROF_STEPS] = P.steps_per_round;
    v[IDL_PROF_CANVAS_PX] = (double)P.canvas_px;
    v[IDL_PROF_IMAGE_PX] = (double)P.image_px;
    v[IDL_PROF_TRIANGLES] = (double)P.n_triangles;
    v[IDL_PROF_PROP_BYTES] = P.prop_bytes;
    for (int i = 0; i < n && i < IDL_PROF_COUNT; ++i) out[i] = v[i];
    IDL_API_END
}

int idl_voronoi(idl_context* ctx, int width, int height, const int32_t* seeds_xy, int64_t n_seeds, int mode,
                int32_t* grid_out, int64_t* passes_out)
{
    IDL_API_BEGIN
    if (!ctx || !grid_out) invalid("arguments must not be NULL");
    check_mode(mode);
    check_dims(width, height, n_seeds);
    check_seed_count(n_seeds);
    if (!seeds_xy) invalid("seeds must not be NULL");
    DeviceGuard g(ctx->device);
    Context& C = *ctx;
    const Canvas cv = make_canvas(width, height);
    upload_seeds(C, seeds_xy, n_seeds, cudaMemcpyHostToDevice);
    int64_t passes = 0;
    const Precleared guard{C};
    clear_for_run(C, cv, width, height, n_seeds, mode == IDL_MODE_REFERENCE && C.direct(), 0, 0);
    sort_seeds_device(C, width, height, n_seeds, 0);
    const bool resolved = start_labels(C, mode, cv, n_seeds, 0, &passes);
    const size_t bytes = (size_t)width * height * 2 * sizeof(int32_t);
    C.outgrid.ensure(bytes);
    auto deliver = [&] {
        dim3 gr(ceil_div(width, 256), height);
        k_compose2<<<gr, 256, 0, C.stream>>>(C.lab[0].as<int32_t>(), cv.pitch, width, height, C.pos.as<uint32_t>(),
                                             C.outgrid.as<int32_t>());
        IDL_LAUNCH();
        IDL_CUDA(cudaMemcpyAsync(grid_out, C.outgrid.ptr, bytes, cudaMemcpyDeviceToHost, C.stream));
        if (resolved) C.fetch_scalars();
        else IDL_CUDA(cudaStreamSynchronize(C.stream));
    };
    if (resolved && passes_out) resolve_arrivals(C, cv, C.pos.as<uint32_t>());
    deliver();
    if (resolved && !idl::resolved(C)) {
        passes = run_passes(C, mode, cv, n_seeds);
        deliver();
    } else if (resolved && passes_out) {
        passes = count_passes(C, mode, cv, n_seeds);
    }
    if (passes_out) *passes_out = passes;
    IDL_API_END
}

int idl_triangulate(idl_context* ctx, int width, int height, const int32_t* seeds_xy, int64_t n_seeds,
                    const int32_t* voronoi_grid, int border_padding, int mode, int32_t* grid_out,
                    int64_t* n_triangles_out, float* timings_out, int32_t* padded_grid_out)
{
    IDL_API_BEGIN
    if (!ctx || !grid_out) invalid("arguments must not be NULL");
    check_mode(mode);
    if (width <= 0 || height <= 0) invalid("width and height must be positive");
    check_seed_count(n_seeds);
    if (!seeds_xy) invalid("seeds must not be NULL");
    DeviceGuard g(ctx->device);
    Context& C = *ctx;
    C.have_result = false;
    const int P = resolve_padding(border_padding);
    upload_seeds(C, seeds_xy, n_seeds, cudaMemcpyHostToDevice);
    const size_t bytes = (size_t)width * height * 3 * sizeof(int32_t);
    C.outgrid.ensure(bytes);
    const int64_t nt = run_triangulate(
        C, width, height, n_seeds, voronoi_grid, P, mode, timings_out, C.outgrid.as<int32_t>(), [&](const Canvas& cv) {
            IDL_CUDA(cudaMemcpyAsync(grid_out, C.outgrid.ptr, bytes, cudaMemcpyDeviceToHost, C.stream));
            if (padded_grid_out && P > 0) {
                const size_t pb = (size_t)cv.Wd * cv.Hd * 2 * sizeof(int32_t);
                C.padded.ensure(pb);
                dim3 gp(ceil_div(cv.Wd, 256), cv.Hd);
                k_compose2<<<gp, 256, 0, C.stream>>>(C.lab[0].as<int32_t>(), cv.pitch, cv.Wd, cv.Hd,
                                                     C.pos.as<uint32_t>(), C.padded.as<int32_t>());
                IDL_LAUNCH();
                IDL_CUDA(cudaMemcpyAsync(padded_grid_out, C.padded.ptr, pb, cudaMemcpyDeviceToHost, C.stream));
            }
        });
    if (n_triangles_out) *n_triangles_out = nt;
    IDL_API_END
}

int idl_get_triangle_vertices(idl_context* ctx, int32_t* verts_out, int64_t capacity)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (!ctx->have_result) throw Error(IDL_ERR_STATE, "no triangulation result on this context");
    if (capacity < ctx->last_n_tri) invalid("capacity is smaller than the triangle count");
    if (ctx->last_n_tri == 0) return IDL_OK;
    if (!verts_out) invalid("verts_out must not be NULL");
    DeviceGuard g(ctx->device);
    const int64_t n = ctx->last_n_tri;
    ctx->verts.ensure((size_t)n * 3 * sizeof(int32_t));
    k_tri_vertices<<<(unsigned)((n * 3 + 255) / 256), 256, 0, ctx->stream>>>(ctx->tris.as<int32_t>(), n,
                                                                          ctx->verts.as<int32_t>());
    IDL_LAUNCH();
    IDL_CUDA(cudaMemcpyAsync(verts_out, ctx->verts.ptr, (size_t)n * 3 * sizeof(int32_t), cudaMemcpyDeviceToHost,
                             ctx->stream));
    IDL_CUDA(cudaStreamSynchronize(ctx->stream));
    IDL_API_END
}

int idl_get_triangles(idl_context* ctx, int32_t* tris_out, int64_t capacity)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (!ctx->have_result) throw Error(IDL_ERR_STATE, "no triangulation result on this context");
    if (capacity < ctx->last_n_tri) invalid("capacity is smaller than the triangle count");
    if (ctx->last_n_tri == 0) return IDL_OK;
    if (!tris_out) invalid("tris_out must not be NULL");
    DeviceGuard g(ctx->device);
    IDL_CUDA(cudaMemcpyAsync(tris_out, ctx->tris.ptr, (size_t)ctx->last_n_tri * 5 * sizeof(int32_t),
                             cudaMemcpyDeviceToHost, ctx->stream));
    IDL_CUDA(cudaStreamSynchronize(ctx->stream));
    IDL_API_END
}

int idl_triangulate_device(idl_context* ctx, int width, int height, const int32_t* d_seeds_xy, int64_t n_seeds,
                           int border_padding, int mode, int32_t* d_grid_out, int64_t* n_triangles_out)
{
    IDL_API_BEGIN
    if (!ctx || !d_grid_out || !d_seeds_xy) invalid("arguments must not be NULL");
    check_mode(mode);
    if (width <= 0 || height <= 0) invalid("width and height must be positive");
    check_seed_count(n_seeds);
    DeviceGuard g(ctx->device);
    Context& C = *ctx;
    C.have_result = false;
    const int P = resolve_padding(border_padding);
    upload_seeds(C, d_seeds_xy, n_seeds, cudaMemcpyDeviceToDevice);
    const int64_t nt = run_triangulate(C, width, height, n_seeds, nullptr, P, mode, nullptr, d_grid_out,
                                       [](const Canvas&) {});
    if (n_triangles_out) *n_triangles_out = nt;
    IDL_API_END
}

int idl_triangles_device(idl_context* ctx, const int32_t** d_tris, const int64_t** d_count)
{
    IDL_API_BEGIN
    if (!ctx) invalid("context must not be NULL");
    if (!ctx->have_result) throw Error(IDL_ERR_STATE, "no triangulation result on this context");
    if (d_tris) *d_tris = ctx->tris.as<int32_t>();
    if (d_count) *d_count = &ctx->sc()->n_triangles;
    IDL_API_END
}

}  // extern "C"
