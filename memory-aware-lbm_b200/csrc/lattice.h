// lattice.h -- the device lattice object behind both C interfaces.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include <vector>
#include "kernels.h"

namespace lbgpu {

// Thread-local error state of the C interfaces (LB_ERR_* codes of include/lbgpu.h).
int set_error(int code, const char *fmt, ...);
int cuda_error(cudaError_t e, const char *what);
int last_error();
const char *last_error_string();
void clear_error();

// Device memory of lattices and requests.  Up to kPoolBytes it comes from a pool per device that keeps up to
// 256 MiB of what was given back (a cudaMalloc takes 0.1 ms and more, a cudaFree waits for the whole
// device: beside others a 1024 x 256 FP32 lattice is made and set up in 0.15 ms instead of 0.87 and closed in 0.06
// instead of 0.6; alone 0.5 and 1.2); what it keeps goes back with the last lattice.  Larger
// parts are cudaMalloc's, one a lattice (made and set up in ms, parts apart before: FP32 8192 x 2048 1.15 and 2.3, FP64
// 16384 x 4096 5.7 and 6.3; a pool that has to grow by 2.4 GB takes 13.5).  Usable on
// any stream at once; given back, with its size, after what `s` still does with it.
constexpr size_t kPoolBytes = (size_t)64 << 20;
cudaError_t device_alloc(void **p, size_t bytes, int device);
cudaError_t device_free(void *p, size_t bytes, int device, cudaStream_t s);
// Lattices alive (each calls hold once and drop once): the last one returns what is kept between them, the
// pools' memory and the pinned buffer of read_back.
void memory_hold();
void memory_drop();

enum { FORM_L = 0, FORM_C = 1 };

// CUDA's limit on gridDim.y (kernels that launch one grid row a lattice row or column).
constexpr size_t kMaxGridY = 65535;

struct Lattice {
    int lx = 0, ly = 0;
    int precision = 0;   // LBGPU_F64 / F32 / F16 / BF16
    int scheme = 0;      // LBGPU_PULL / LBGPU_AA
    DevLattice d{};
    size_t elem = 8;     // bytes per stored population
    int cur = 0;         // buffer holding the state
    int form = FORM_L;   // see kernels.cu
    int pending = 0;     // form C only: 1 when the post-stream state is the current one
    long long n = 0;     // index of the last collision (form C) or of the state (form L)
    bool ghosts = false; // keep the ghost ring exact (drop-in interface)
    bool zgb_each_step = false;  // native: extrapolated outlet before every step
    int sweep_steps = 1;         // lbgpu_set_sweep_steps (runs of pull steps share launches either way)
    cudaStream_t stream = nullptr;
    size_t bytes = 0;
    void *memory = nullptr;        // the one allocation that d's pointers lead into
    size_t memory_bytes = 0;
    bool held = false;             // counted by memory_hold
    bool keep_roles = false;       // a caller captured the stream: an even number of steps leaves buffers and slots in place
    int launches = 0;    // kernels launched by the last public call
    unsigned long long h2d_bytes = 0, d2h_bytes = 0;  // bytes copied host<->device so far
    int device = 0;      // CUDA device the lattice lives on

    std::vector<double> bc_host;   // [16*nb] last uploaded boundary tables
    std::vector<int> zgb_src_host; // [4*nb]
    double *stage = nullptr;       // device staging for record transfers
    size_t stage_bytes = 0;

    int create(int lx, int ly, int precision, int scheme);
    void destroy();
    void reset_roles();
    int see_capture(bool &capturing);

    // per-step operations (asynchronous on `stream`)
    int op_collide();        // collide the current state in place or through the pull kernel
    int op_propagate();      // mark (or perform) the stream
    int materialize();       // form C + pending -> form L
    int zgb_pass();          // extrapolated outlet densities into the tables (zgb_src slots)
    int aa_step();           // one AA time step (even or odd kernel)
    int step(int nsteps);    // full native steps
    void view(int &v, int &par) const;  // read-out view and stale side parity of the state
    long long steps_done() const;

    // data movement
    int upload_bc(const double *bc);      // host [16*nb]
    int upload_bc_range(const double *bc, size_t lo, size_t hi);  // entries lo..hi-1 of them, without waiting
    int upload_zgb_src(const int *src);   // host [4*nb]
    // host tag[X*(ly+2)+Y], validated here; zgb_row: rows of the extrapolated outlet, or null
    int upload_tags(const uint8_t *tag_xy, const uint8_t *zgb_row);
    int upload_records(int b, const double *host, int rs, int X0, int X1);
    // rows Y0..Y0+H-1 of columns X0..X1-1 from host records laid out like upload_records' (host
    // points at column X0, row 0)
    int upload_record_rows(int b, const double *host, int rs, int X0, int X1, int Y0, int H);
    // the stale-slot and ghost-ring sources of buffer b only: columns 0, 1, lx, lx+1 and rows
    // 0, 1, ly, ly+1 (the pull kernel writes the rest before anything reads it)
    int upload_records_edges(int b, const double *host, int rs);
    int upload_tags_xy(const uint8_t *tag_xy);   // host order, already validated
    int readout_records(double *host, int rs, const uint64_t *dynp_dev, int X0, int X1);
    int readout_populations(double *host);       // [lx+2][ly+2][9] into a pageable array
    int init_side_from(int b, int par);
    int init_cylinder(double umax);  // equilibrium Poiseuille populations into the current buffer
    int get_macros(double *rho, double *ux, double *uy);  // host [ly][lx] arrays
    int moments(double out[8]);                           // FP64 sums (kernels.h)
    int velocity_accumulate();
    int velocity_average(double *ux, double *uy, long long *samples);
    double *red_scratch = nullptr;  // (ly+2)*8 partial sums + 8 results
    double *vel_acc = nullptr;      // 2*lx*ly running velocity sums
    float *shift = nullptr;         // 16-bit storage: per-row shift velocity [ly+2] (d.g.shift_u)
    bool rs = false;                // 16-bit storage: stochastic rounding of stored values
    unsigned rs_seed = 0;
    // the key of collision k into d.g before a collision launch
    void set_rs_keys(long long k);
    // the host's side of a tile launch of T steps: slots and rings change roles (kernels.h launch_tile)
    void after_tile(int T);
    long long vel_samples = 0;
    int check(const char *what);   // cudaGetLastError -> error code
    int side_par_stale() const { return (int)((n + 1) & 1); }
    size_t stage_cols(int rs) const;
    int ensure_stage(size_t bytes_needed);
};

}  // namespace lbgpu

// The opaque handle of include/lbgpu.h.
struct lbgpu_lattice {
    lbgpu::Lattice L;
};
