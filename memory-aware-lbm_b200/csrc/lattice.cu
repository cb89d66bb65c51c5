// lattice.cu -- allocation, state machine and data movement of a device lattice.
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include "codec.cuh"
#include "lattice.h"
#include "readback.h"
#include "lbgpu.h"

namespace lbgpu {

// ---- thread-local error state ---------------------------------------------------------
namespace {
thread_local int g_err = 0;
thread_local char g_msg[512] = "";
}  // namespace

int set_error(int code, const char *fmt, ...)
{
    if (g_err == 0) {  // keep the first error until cleared
        g_err = code;
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(g_msg, sizeof g_msg, fmt, ap);
        va_end(ap);
    }
    return code;
}

int cuda_error(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return LB_OK;
    if (e == cudaErrorMemoryAllocation)
        return set_error(LB_ERR_ALLOC, "%s: %s", what, cudaGetErrorString(e));
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver)
        return set_error(LB_ERR_NO_DEVICE, "%s: %s", what, cudaGetErrorString(e));
    return set_error(LB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int last_error() { return g_err; }
const char *last_error_string() { return g_msg; }
void clear_error() { g_err = 0; g_msg[0] = 0; }

// ---- device memory ---------------------------------------------------------------------
namespace {
constexpr int kPools = 64;
struct Pool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
};
std::mutex g_mem_mu;
Pool g_pool[kPools];
int g_lattices = 0;

cudaError_t pool_of(int device, Pool &p)
{
    if (device < 0 || device >= kPools) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_mem_mu);
    Pool &own = g_pool[device];
    if (!own.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        if (cudaError_t e = cudaMemPoolCreate(&own.pool, &props)) return e;
        unsigned long long keep = 256ull << 20;
        cudaMemPoolSetAttribute(own.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    if (!own.stream)
        if (cudaError_t e = cudaStreamCreateWithFlags(&own.stream, cudaStreamNonBlocking)) return e;
    p = own;
    return cudaSuccess;
}
}  // namespace

// A pool's allocations and frees run on a stream of its own, which no lattice's work touches: CUDA follows the
// events between streams that have allocated, and a batch of 256 members, each with its stream, then spent
// 600 us a call on them where it takes 115 (one B200, two FP32 steps of 100 x 60 members).
cudaError_t device_alloc(void **p, size_t bytes, int device)
{
    *p = nullptr;
    if (bytes > kPoolBytes) return cudaMalloc(p, bytes);
    Pool pool;
    if (cudaError_t e = pool_of(device, pool)) return e;
    if (cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool.pool, pool.stream)) return e;
    return cudaStreamSynchronize(pool.stream);
}

cudaError_t device_free(void *p, size_t bytes, int device, cudaStream_t s)
{
    if (bytes > kPoolBytes) return cudaFree(p);
    Pool pool;
    if (cudaError_t e = pool_of(device, pool)) return e;
    const cudaError_t e = cudaStreamSynchronize(s);
    const cudaError_t f = cudaFreeAsync(p, pool.stream);
    // (the wait is where the pool gives back what it keeps too much of, and where cudaMalloc can have the rest)
    const cudaError_t g = cudaStreamSynchronize(pool.stream);
    return e ? e : (f ? f : g);
}

void memory_hold()
{
    std::lock_guard<std::mutex> lock(g_mem_mu);
    ++g_lattices;
}

void memory_drop()
{
    std::lock_guard<std::mutex> lock(g_mem_mu);
    if (--g_lattices > 0) return;
    for (Pool &p : g_pool) {     // (destroyed, not trimmed: a device reset in between is then harmless)
        if (p.stream) {
            cudaStreamSynchronize(p.stream);
            cudaStreamDestroy(p.stream);
        }
        if (p.pool) cudaMemPoolDestroy(p.pool);
        p = Pool{};
    }
    read_back_release();
}

#define LB_TRY(expr)                                \
    do {                                            \
        int rc_ = (expr);                           \
        if (rc_ != LB_OK) return rc_;               \
    } while (0)
#define LB_CUDA(call, what) LB_TRY(cuda_error((call), (what)))

// ---- lifetime -------------------------------------------------------------------------
static size_t elem_bytes(int precision)
{
    switch (precision) {
    case LBGPU_F64: return 8;
    case LBGPU_F32: return 4;
    default: return 2;
    }
}

int Lattice::create(int lx_, int ly_, int precision_, int scheme_)
{
    // The row-wise kernels launch one grid row per lattice row, ghost rows included, and CUDA
    // caps gridDim.y at 65535: hence ly <= LBGPU_MAX_LY.
    if (lx_ < 1 || ly_ < 1 || lx_ > LBGPU_MAX_LX || ly_ > LBGPU_MAX_LY)
        return set_error(LB_ERR_ARG, "lattice size %d x %d out of range (1..%d x 1..%d)", lx_, ly_,
                         LBGPU_MAX_LX, LBGPU_MAX_LY);
    if (precision_ < LBGPU_F64 || precision_ > LBGPU_BF16)
        return set_error(LB_ERR_ARG, "unknown precision %d", precision_);
    if (scheme_ != LBGPU_PULL && scheme_ != LBGPU_AA)
        return set_error(LB_ERR_ARG, "unknown scheme %d", scheme_);
    lx = lx_; ly = ly_; precision = precision_; scheme = scheme_;
    elem = elem_bytes(precision);
    d.g = make_geo(lx, ly, (int)elem);
    d.precision = precision;
    d.omega = 1.0;
    d.scale = 1.0f; d.inv_scale = 1.0f;
    int ndev = 0;
    LB_CUDA(cudaGetDeviceCount(&ndev), "cudaGetDeviceCount");
    if (ndev == 0) return set_error(LB_ERR_NO_DEVICE, "no CUDA device");
    LB_CUDA(cudaGetDevice(&device), "cudaGetDevice");
    LB_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");

    // One allocation for everything, its parts on 256-byte boundaries, and those of a page of 2 MiB or more on a page's
    // (BF16 700 x 200, single steps, one B200: 8.9 us instead of 9.7); all zero but the slots without an
    // extrapolated row.
    const size_t nbuf = (scheme == LBGPU_AA) ? 1 : 2;
    const size_t pbytes = 9 * (size_t)d.g.plane * elem;
    const size_t sbytes = (size_t)side_slots(precision, scheme) * 9 * (size_t)d.g.nper * elem;
    const size_t gbytes = scheme == LBGPU_AA ? 9 * (size_t)d.g.nghost() * elem : 0;
    const size_t part[8] = {pbytes, nbuf == 2 ? pbytes : 0, gbytes, sbytes, (size_t)d.g.plane,
                            16 * (size_t)d.g.nb * sizeof(double), 2 * (size_t)(ly + 2) * sizeof(double),
                            4 * (size_t)d.g.nb * sizeof(int)};
    size_t at[9] = {0};
    for (int k = 0; k < 8; ++k) {
        const size_t page = (size_t)2 << 20;
        if (part[k] >= page) at[k] = (at[k] + page - 1) / page * page;
        at[k + 1] = at[k] + (part[k] + 255) / 256 * 256;
        bytes += part[k];
    }
    memory_hold();
    held = true;
    memory_bytes = at[8];
    LB_CUDA(device_alloc(&memory, memory_bytes, device), "device memory (lattice)");
    char *m = static_cast<char *>(memory);
    LB_CUDA(cudaMemsetAsync(m, 0, at[7], stream), "cudaMemset(lattice)");
    LB_CUDA(cudaMemsetAsync(m + at[7], 0xff, part[7], stream), "cudaMemset(zgb slots)");
    d.buf[0] = m + at[0];
    d.buf[1] = nbuf == 2 ? m + at[1] : nullptr;
    d.ghost2 = gbytes ? m + at[2] : nullptr;
    d.side = m + at[3];
    d.tag = reinterpret_cast<const uint8_t *>(m + at[4]);
    d.bc = reinterpret_cast<double *>(m + at[5]);
    d.zrho = reinterpret_cast<double *>(m + at[6]);
    d.zgb_src = reinterpret_cast<const int *>(m + at[7]);
    reset_roles();
    bc_host.assign(16 * (size_t)d.g.nb, 0.0);
    zgb_src_host.assign(4 * (size_t)d.g.nb, -1);
    return check("lattice create");
}

// The state is written afresh, into buffer `cur`: each parity's stale slots in its own slot, each ring in its
// buffer; or where a captured graph expects it, whose steps then start from the same buffers and slots
// again after as many steps as before its capture.
void Lattice::reset_roles()
{
    cur = keep_roles ? cur ^ (int)(n & 1) : 0;
    if (!keep_roles) {
        d.side_slot[0] = 0;
        d.side_slot[1] = 1;
    }
    d.ghost_flip = 0;
    form = FORM_L; pending = 0; n = 0;
}

// Whether the caller captures the stream; remembered, because its graph holds the buffers and slots of now.
int Lattice::see_capture(bool &capturing)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    LB_CUDA(cudaStreamIsCapturing(stream, &status), "cudaStreamIsCapturing");
    capturing = status != cudaStreamCaptureStatusNone;
    keep_roles = keep_roles || capturing;
    return LB_OK;
}

void Lattice::destroy()
{
    if (stream) cudaStreamSynchronize(stream);
    if (memory) device_free(memory, memory_bytes, device, stream);
    memory = nullptr;
    if (stage) device_free(stage, stage_bytes, device, stream);
    if (red_scratch) cudaFree(red_scratch);
    if (vel_acc) cudaFree(vel_acc);
    if (shift) cudaFree(shift);
    red_scratch = nullptr; vel_acc = nullptr; vel_samples = 0; shift = nullptr;
    if (stream) cudaStreamDestroy(stream);
    if (held) memory_drop();
    held = false;
    d = DevLattice{};
    stage = nullptr; stage_bytes = 0; stream = nullptr;
}

int Lattice::check(const char *what)
{
    return cuda_error(cudaGetLastError(), what);
}

// How the post-stream state is read, and which side parity holds its stale slots.
void Lattice::view(int &v, int &par) const
{
    if (scheme == LBGPU_AA) {
        if (form == FORM_L) { v = VIEW_AA_NATURAL; par = (int)(n & 1); }
        else { v = VIEW_AA_SWAPPED; par = (int)((n + 1) & 1); }
        return;
    }
    par = (int)((n + 1) & 1);
    v = (form == FORM_C && pending) ? VIEW_PULL_PENDING : VIEW_DIRECT;
}

// Collision k produces the post-collision state C_k; its stored values round with key k.
void Lattice::set_rs_keys(long long k)
{
    d.g.rs_key = rs ? rs_key(rs_seed, (unsigned long long)k) : 0u;
}

// ---- state machine (pull scheme) ------------------------------------------------------
int Lattice::op_collide()
{
    if (scheme != LBGPU_PULL) return set_error(LB_ERR_STATE, "collide/propagate need the pull scheme");
    if (form == FORM_C && pending) {
        set_rs_keys(n + 1);
        launch_pull(d, cur, (int)((n + 1) & 1), ghosts, stream);
        launches += pull_launches(d, ghosts) - 1;
        cur = 1 - cur;
        ++n;
    } else {
        set_rs_keys(n);
        launch_collide_inplace(d, cur, (int)(n & 1), stream);
        form = FORM_C;
    }
    pending = 0;
    ++launches;
    return check("collide");
}

int Lattice::materialize()
{
    if (scheme != LBGPU_PULL) return set_error(LB_ERR_STATE, "materialize needs the pull scheme");
    if (form == FORM_C && pending) {
        launch_stream(d, cur, (int)((n + 1) & 1), stream);
        cur = 1 - cur;
        ++n;
        form = FORM_L;
        pending = 0;
        ++launches;
    }
    return check("stream");
}

int Lattice::op_propagate()
{
    if (scheme != LBGPU_PULL) return set_error(LB_ERR_STATE, "collide/propagate need the pull scheme");
    if (form == FORM_C && !pending) {
        pending = 1;
        return LB_OK;
    }
    LB_TRY(materialize());
    // stream of an uncollided state: it acts as its own post-collision state
    launch_side_from_buf(d, cur, (int)(n & 1), stream);
    ++launches;
    form = FORM_C;
    pending = 1;
    return check("propagate");
}

int Lattice::zgb_pass()
{
    if (lx < 2) return set_error(LB_ERR_ARG, "the extrapolated outlet needs lx >= 2");
    if (scheme == LBGPU_PULL && form == FORM_C && !pending)
        return set_error(LB_ERR_STATE, "extrapolated outlet requested on a collided state");
    int v, par;
    view(v, par);
    launch_zgb(d, v, cur, par, stream);
    ++launches;
    return check("zgb pass");
}

// One AA time step: natural form -> even kernel (C_m into the opposite slots); swapped form ->
// odd kernel (gather, collide, scatter), leaving the natural form two steps on.
int Lattice::aa_step()
{
    if (form == FORM_L) {
        set_rs_keys(n);
        launch_aa_even(d, (int)(n & 1), stream);
        form = FORM_C;
        pending = 1;
    } else {
        set_rs_keys(n + 1);
        launch_aa_odd(d, (int)((n + 1) & 1), stream);
        n += 2;
        form = FORM_L;
        pending = 0;
    }
    ++launches;
    return check("aa step");
}

int Lattice::step(int nsteps)
{
    if (nsteps < 0) return set_error(LB_ERR_ARG, "negative step count");
    launches = 0;
    // A single step turns the buffers over, so an even number of them leaves them in place, and a caller's graph
    // of them can be replayed; a tile launch turns them over too, whatever its steps.  So steps stay single
    // while the caller captures the stream, and from then on tiles go in pairs of equal launches, which
    // leave the buffers and the side store's slots where they were.
    bool capturing = false;
    if (nsteps > 0) LB_TRY(see_capture(capturing));
    int second = 0;       // steps of a pair's second launch
    for (int s = 0; s < nsteps; ++s) {
        // a run of pull steps: several a launch, the state as single steps leave it
        if (scheme == LBGPU_PULL && !ghosts && form == FORM_C && pending && !capturing) {
            const int rest = nsteps - s;
            if (const int T = second ? second : tile_steps(d, keep_roles ? rest / 2 : rest, zgb_each_step, rs)) {
                second = keep_roles && !second ? T : 0;
                unsigned keys[8] = {0};
                for (int k = 0; rs && k < T; ++k) keys[k] = rs_key(rs_seed, (unsigned long long)(n + 1 + k));
                launch_tile(d, cur, (int)(n & 1), T, zgb_each_step, keys, stream);
                after_tile(T);
                s += T - 1;
                ++launches;
                LB_TRY(check("tile steps"));
                continue;
            }
        }
        if (zgb_each_step) LB_TRY(zgb_pass());
        if (scheme == LBGPU_AA) {
            LB_TRY(aa_step());
        } else {
            LB_TRY(op_collide());
            LB_TRY(op_propagate());
        }
    }
    return LB_OK;
}

void Lattice::after_tile(int T)
{
    const int a = (int)((n + 1) & 1);
    d.side_slot[a] = side_other(d, a);
    if (d.g.shift_u) d.side_slot[1 - a] = side_other(d, 1 - a);
    d.ghost_flip ^= 1;
    cur = 1 - cur;
    n += T;
}

long long Lattice::steps_done() const
{
    if (form == FORM_C && pending) return n + 1;
    return n;
}

// Results up to this size are copied from a device buffer; larger ones go through read_back.  us a call on one B200, buffer
// and read_back: fields 400 x 90 (0.9 MB) 109 and -, 400 x 120 (1.2 MB) 129 and 103; velocity averages 250 x 51 48 and
// 102; populations, whose chunks of columns are transposed, 600 x 150 (6.7 MB) 365 and 461, 700 x 200 (10 MB) 537
// and 424.
static constexpr size_t kStagedBytes = (size_t)1 << 20, kStagedPops = (size_t)8 << 20;

// ---- data movement --------------------------------------------------------------------
int Lattice::ensure_stage(size_t need)
{
    if (stage_bytes >= need) return LB_OK;
    if (stage) { device_free(stage, stage_bytes, device, stream); stage = nullptr; stage_bytes = 0; }
    void *p = nullptr;
    LB_CUDA(device_alloc(&p, need, device), "device memory (staging)");
    stage = static_cast<double *>(p);
    stage_bytes = need;
    return LB_OK;
}

size_t Lattice::stage_cols(int rs) const
{
    const size_t col = (size_t)(ly + 2) * rs * sizeof(double);
    size_t cols = ((size_t)64 << 20) / col;
    if (cols < 1) cols = 1;
    if (cols > (size_t)(lx + 2)) cols = (size_t)(lx + 2);
    if (cols > kMaxGridY) cols = kMaxGridY;   // one grid row a column in the copy kernels
    return cols;
}

int Lattice::upload_records(int b, const double *host, int rs, int X0, int X1)
{
    const size_t col = (size_t)(ly + 2) * rs;
    const size_t cols = stage_cols(rs);
    LB_TRY(ensure_stage(cols * col * sizeof(double)));
    for (int c0 = X0; c0 < X1; c0 += (int)cols) {
        const int c1 = (c0 + (int)cols < X1) ? c0 + (int)cols : X1;
        LB_CUDA(cudaMemcpyAsync(stage, host + (size_t)(c0 - X0) * col,
                                (size_t)(c1 - c0) * col * sizeof(double),
                                cudaMemcpyHostToDevice, stream), "upload populations");
        h2d_bytes += (size_t)(c1 - c0) * col * sizeof(double);
        launch_upload(d, b, stage, rs, c0, c1, 0, ly + 2, stream);
        ++launches;
    }
    return check("upload");
}

int Lattice::upload_record_rows(int b, const double *host, int rs, int X0, int X1, int Y0, int H)
{
    if (X1 <= X0 || H <= 0) return LB_OK;
    const size_t col = (size_t)(ly + 2) * rs, band = (size_t)H * rs;
    size_t cols = ((size_t)64 << 20) / (band * sizeof(double));
    if (cols < 1) cols = 1;
    if (cols > (size_t)(X1 - X0)) cols = (size_t)(X1 - X0);
    if (cols > kMaxGridY) cols = kMaxGridY;
    LB_TRY(ensure_stage(cols * band * sizeof(double)));
    for (int c0 = X0; c0 < X1; c0 += (int)cols) {
        const int c1 = (c0 + (int)cols < X1) ? c0 + (int)cols : X1;
        LB_CUDA(cudaMemcpy2DAsync(stage, band * sizeof(double), host + (size_t)(c0 - X0) * col + (size_t)Y0 * rs,
                                  col * sizeof(double), band * sizeof(double), (size_t)(c1 - c0),
                                  cudaMemcpyHostToDevice, stream), "upload population rows");
        h2d_bytes += (size_t)(c1 - c0) * band * sizeof(double);
        launch_upload(d, b, stage, rs, c0, c1, Y0, H, stream);
        ++launches;
    }
    return check("upload rows");
}

int Lattice::upload_records_edges(int b, const double *host, int rs)
{
    if (lx < 4 || ly < 4) return upload_records(b, host, rs, 0, lx + 2);
    const size_t col = (size_t)(ly + 2) * rs;
    LB_TRY(upload_records(b, host, rs, 0, 2));
    LB_TRY(upload_records(b, host + (size_t)lx * col, rs, lx, lx + 2));
    LB_TRY(upload_record_rows(b, host + 2 * col, rs, 2, lx, 0, 2));
    return upload_record_rows(b, host + 2 * col, rs, 2, lx, ly, 2);
}

int Lattice::readout_records(double *host, int rs, const uint64_t *dynp_dev, int X0, int X1)
{
    const size_t col = (size_t)(ly + 2) * rs;
    const size_t cols = stage_cols(rs);
    LB_TRY(ensure_stage(cols * col * sizeof(double)));
    int v, par;
    view(v, par);
    for (int c0 = X0; c0 < X1; c0 += (int)cols) {
        const int c1 = (c0 + (int)cols < X1) ? c0 + (int)cols : X1;
        launch_readout(d, v, cur, par, c0, c1, stage, rs, dynp_dev, stream);
        ++launches;
        LB_CUDA(cudaMemcpyAsync(host + (size_t)(c0 - X0) * col, stage,
                                (size_t)(c1 - c0) * col * sizeof(double),
                                cudaMemcpyDeviceToHost, stream), "download populations");
        d2h_bytes += (size_t)(c1 - c0) * col * sizeof(double);
    }
    LB_CUDA(cudaStreamSynchronize(stream), "readout");
    return check("readout");
}

int Lattice::readout_populations(double *host)
{
    // small ones through the device staging: pinned memory that nobody holds yet takes 1.7 ms to get
    if ((size_t)(lx + 2) * (ly + 2) * 72 <= kStagedPops) return readout_records(host, 9, nullptr, 0, lx + 2);
    int v, par;
    view(v, par);
    const size_t col = (size_t)(ly + 2) * 9;
    const cudaError_t e = read_back(
        device, stream, lx + 2, col * sizeof(double),
        [&](long long x0, long long x1, double *dst) {
            launch_readout(d, v, cur, par, (int)x0, (int)x1, dst, 9, nullptr, stream);
        },
        [&](long long x0, long long x1, const double *src) {
            std::memcpy(host + (size_t)x0 * col, src, (size_t)(x1 - x0) * col * sizeof(double));
        });
    d2h_bytes += (size_t)(lx + 2) * col * sizeof(double);
    return cuda_error(e, "readout");
}

int Lattice::init_side_from(int b, int par)
{
    launch_side_from_buf(d, b, par, stream);
    ++launches;
    return check("side store init");
}

int Lattice::init_cylinder(double umax)
{
    launch_init_cylinder(d, cur, umax, stream);
    ++launches;
    return check("init cylinder");
}

int Lattice::get_macros(double *rho, double *ux, double *uy)
{
    int v, par;
    view(v, par);
    double *const to[3] = {rho, ux, uy};
    int n = 0;
    double *field[3];
    for (double *p : to)
        if (p) field[n++] = p;
    const size_t nn = (size_t)lx * ly;
    if (n && n * nn * sizeof(double) <= kStagedBytes) {
        LB_TRY(ensure_stage(3 * nn * sizeof(double)));
        launch_macros(d, v, cur, par, 1, ly + 1, stage, stage + nn, stage + 2 * nn, stream);
        LB_TRY(check("macros"));
        for (int j = 0; j < 3; ++j)
            if (to[j])
                LB_CUDA(cudaMemcpyAsync(to[j], stage + j * nn, nn * sizeof(double), cudaMemcpyDeviceToHost, stream), "macros");
        d2h_bytes += n * nn * sizeof(double);
        return cuda_error(cudaStreamSynchronize(stream), "macros");
    }
    // one item a row: its values of each field wanted, one field after the other in a chunk
    const cudaError_t e = read_back(
        device, stream, n ? ly : 0, (size_t)n * lx * sizeof(double),
        [&](long long y0, long long y1, double *dst) {
            const size_t m = (size_t)(y1 - y0) * lx;
            double *at[3];
            int k = 0;
            for (int j = 0; j < 3; ++j) at[j] = to[j] ? dst + m * k++ : nullptr;
            launch_macros(d, v, cur, par, (int)y0 + 1, (int)y1 + 1, at[0], at[1], at[2], stream);
        },
        [&](long long y0, long long y1, const double *src) {
            const size_t m = (size_t)(y1 - y0) * lx;
            for (int k = 0; k < n; ++k) std::memcpy(field[k] + (size_t)y0 * lx, src + m * k, m * sizeof(double));
        });
    d2h_bytes += (size_t)n * lx * ly * sizeof(double);
    return cuda_error(e, "macros");
}

int Lattice::moments(double out[8])
{
    if (!red_scratch) {
        void *p = nullptr;
        LB_CUDA(cudaMalloc(&p, ((size_t)(ly + 2) * 8 + 8) * sizeof(double)), "cudaMalloc(reduction)");
        red_scratch = static_cast<double *>(p);
    }
    int v, par;
    view(v, par);
    double *res = red_scratch + (size_t)(ly + 2) * 8;
    launch_moments(d, v, cur, par, red_scratch, res, stream);
    LB_TRY(check("moments"));
    LB_CUDA(cudaMemcpyAsync(out, res, 8 * sizeof(double), cudaMemcpyDeviceToHost, stream), "moments");
    d2h_bytes += 8 * sizeof(double);
    LB_CUDA(cudaStreamSynchronize(stream), "moments");
    return LB_OK;
}

int Lattice::velocity_accumulate()
{
    const size_t bytes = 2 * (size_t)lx * ly * sizeof(double);
    if (!vel_acc) {
        void *p = nullptr;
        LB_CUDA(cudaMalloc(&p, bytes), "cudaMalloc(velocity sums)");
        vel_acc = static_cast<double *>(p);
        LB_CUDA(cudaMemsetAsync(vel_acc, 0, bytes, stream), "clear velocity sums");
        vel_samples = 0;
    }
    bool capturing;
    LB_TRY(see_capture(capturing));
    int v, par;
    view(v, par);
    launch_accumulate_velocity(d, v, cur, par, vel_acc, stream);
    ++vel_samples;
    return check("velocity accumulate");
}

int Lattice::velocity_average(double *ux, double *uy, long long *samples)
{
    const size_t nn = (size_t)lx * ly;
    if (samples) *samples = vel_samples;
    if (!vel_acc || vel_samples == 0) return set_error(LB_ERR_STATE, "no velocity samples accumulated");
    const double k = 1.0 / (double)vel_samples;
    double *const to[2] = {ux, uy};
    if (2 * nn * sizeof(double) <= kStagedBytes) {
        // small: copied from a device buffer, or the smallest as they are and scaled here (20 x 16 27 us instead of 32)
        const bool here = nn <= 4096;
        const double *from = vel_acc;
        if (!here) {
            LB_TRY(ensure_stage(2 * nn * sizeof(double)));
            launch_scaled(vel_acc, k, stage, 2 * (long long)nn, stream);
            LB_TRY(check("velocity average"));
            from = stage;
        }
        for (int j = 0; j < 2; ++j)
            if (to[j]) {
                LB_CUDA(cudaMemcpyAsync(to[j], from + j * nn, nn * sizeof(double), cudaMemcpyDeviceToHost, stream), "velocity average");
                d2h_bytes += nn * sizeof(double);
            }
        LB_CUDA(cudaStreamSynchronize(stream), "velocity average");
        if (here)
            for (double *p : to)
                for (size_t x = 0; p && x < nn; ++x) p[x] *= k;
        return LB_OK;
    }
    for (int j = 0; j < 2; ++j) {
        if (!to[j]) continue;
        const cudaError_t e = read_back(
            device, stream, ly, (size_t)lx * sizeof(double),
            [&](long long y0, long long y1, double *dst) {
                launch_scaled(vel_acc + (size_t)j * nn + (size_t)y0 * lx, k, dst, (y1 - y0) * lx, stream);
            },
            [&](long long y0, long long y1, const double *src) {
                std::memcpy(to[j] + (size_t)y0 * lx, src, (size_t)(y1 - y0) * lx * sizeof(double));
            });
        LB_CUDA(e, "velocity average");
        d2h_bytes += nn * 8;
    }
    return LB_OK;
}

int Lattice::upload_bc(const double *bc)
{
    std::memcpy(bc_host.data(), bc, bc_host.size() * sizeof(double));
    LB_CUDA(cudaMemcpyAsync(d.bc, bc_host.data(), bc_host.size() * sizeof(double),
                            cudaMemcpyHostToDevice, stream), "upload tables");
    h2d_bytes += bc_host.size() * sizeof(double);
    // the copy reads bc_host asynchronously: wait so the caller may reuse its array and
    // the next refresh may overwrite bc_host
    LB_CUDA(cudaStreamSynchronize(stream), "upload tables");
    return LB_OK;
}

int Lattice::upload_bc_range(const double *bc, size_t lo, size_t hi)
{
    if (hi <= lo) return LB_OK;
    std::memcpy(bc_host.data() + lo, bc + lo, (hi - lo) * sizeof(double));
    // a copy from pageable memory has taken its source when the call returns, so nothing waits here
    LB_CUDA(cudaMemcpyAsync(d.bc + lo, bc_host.data() + lo, (hi - lo) * sizeof(double), cudaMemcpyHostToDevice,
                            stream), "upload tables");
    h2d_bytes += (hi - lo) * sizeof(double);
    return LB_OK;
}

int Lattice::upload_zgb_src(const int *src)
{
    std::memcpy(zgb_src_host.data(), src, zgb_src_host.size() * sizeof(int));
    LB_CUDA(cudaMemcpyAsync(const_cast<int *>(d.zgb_src), zgb_src_host.data(),
                            zgb_src_host.size() * sizeof(int), cudaMemcpyHostToDevice, stream),
            "upload zgb slots");
    h2d_bytes += zgb_src_host.size() * sizeof(int);
    LB_CUDA(cudaStreamSynchronize(stream), "upload zgb slots");
    return LB_OK;
}

int Lattice::upload_tags(const uint8_t *tag_xy, const uint8_t *zgb_row)
{
    int inside = 0, outlet = lx >= 4;
    long long rows = 0;
    for (int X = 0; X < lx + 2; ++X)
        for (int Y = 0; Y < ly + 2; ++Y) {
            const int t = tag_xy[(size_t)X * (ly + 2) + Y];
            if (t >= LBGPU_NUM_TAGS)
                return set_error(LB_ERR_ARG, "tag %d at (%d,%d) out of range", t, X, Y);
            if (d.g.interior(X, Y) && t == LBGPU_TAG_NONE)
                return set_error(LB_ERR_DYNAMICS, "interior node (%d,%d) has no dynamics", X, Y);
            if (t >= LBGPU_TAG_UPPER_ZOUHE && X > 1 && X < lx && Y > 1 && Y < ly) inside = 1;
            if (t >= LBGPU_TAG_UPPER_ZOUHE && (Y == 1 || Y == ly)) ++rows;
            // an extrapolated row's pressure nodes anywhere but at its end, or the rows at the walls
            const bool right = t == LBGPU_TAG_RIGHT_PRESSURE_ZOUHE || t == LBGPU_TAG_RIGHT_PRESSURE_REGULARIZED;
            if (zgb_row && zgb_row[Y] && right && (X != lx || Y < 2 || Y > ly - 1)) outlet = 0;
        }
    LB_TRY(upload_tags_xy(tag_xy));
    d.rules_inside = inside;
    d.row_rules = rows > lx;
    d.outlet_tiles = outlet;
    return LB_OK;
}

// The host array in its own order to the device, transposed there (a host transpose writes one
// byte a cache line).
int Lattice::upload_tags_xy(const uint8_t *tag_xy)
{
    const size_t n = (size_t)(lx + 2) * (ly + 2);
    LB_TRY(ensure_stage(n));
    LB_CUDA(cudaMemcpyAsync(stage, tag_xy, n, cudaMemcpyHostToDevice, stream), "upload tags");
    h2d_bytes += n;
    launch_tags_from_xy(d, reinterpret_cast<const uint8_t *>(stage), stream);
    LB_TRY(check("tags"));
    LB_CUDA(cudaStreamSynchronize(stream), "upload tags");
    return LB_OK;
}

}  // namespace lbgpu
