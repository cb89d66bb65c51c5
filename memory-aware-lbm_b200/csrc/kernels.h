// kernels.h -- host launchers of the device kernels (all asynchronous on `s`).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "layout.cuh"
#include "lbgpu.h"

namespace lbgpu {

// Device-side view of one lattice's data, passed by value to the launchers.
struct DevLattice {
    Geo g;
    int precision;       // LBGPU_F64 / F32 / F16 / BF16: element type of buf and side
    void *buf[2];        // population buffers (buf[1] unused by the AA scheme)
    void *side;          // stale-slot store: side_slots() slots of [9][nper]
    int side_slot[2];    // the slot of each collision parity
    int ghost_flip;      // 1: the ring that belongs to the second buffer is in the current one (launch_tile)
    int rules_inside;    // some node off the perimeter has a boundary rule
    int row_rules;       // more than half of the first and last rows' nodes have boundary rules
    int outlet_tiles;    // the extrapolated outlet's nodes lie where the tile kernel extrapolates them
    void *ghost2;        // AA only: the second buffer's ghost ring [9][nghost] (see logical_at())
    const uint8_t *tag;  // tag plane
    double *bc;          // boundary tables [8][2][nb]
    const int *zgb_src;  // [4][nb]: pressure-table slot -> source row of its ZGB density, or -1
    double *zrho;        // [2*(ly+2)]: rho(lx-1, Y), rho(lx-2, Y) of the last ZGB pass
    double omega;
    float scale, inv_scale;  // FP16/BF16 offset storage: stored = (f - w) * scale
};

// The side store's slots: AA two; pull three (FP64, FP32), or four for 16-bit storage, whose row-shifted tiles write both
// parities' slots beside those they read.
inline int side_slots(int precision, int scheme)
{
    return scheme == LBGPU_AA ? 2 : (precision == LBGPU_F64 || precision == LBGPU_F32 ? 3 : 4);
}
// The slot that a tile launch writes for parity p beside the one in use; the next launch from the same parity takes
// that one back, so that two launches leave the slots where they were.
inline int side_other(const DevLattice &d, int p)
{
    return d.precision == LBGPU_F64 || d.precision == LBGPU_F32 ? 3 - d.side_slot[0] - d.side_slot[1] : d.side_slot[p] ^ 2;
}

// How the post-stream state is read from a buffer:
//   VIEW_DIRECT        the buffer holds it (pull form L, or a collided state read as is)
//   VIEW_PULL_PENDING  the buffer holds C_n; the state is C_n streamed (side store: C_{n-1})
//   VIEW_AA_NATURAL    AA buffer in natural slots; stale slots in the side store
//   VIEW_AA_SWAPPED    AA buffer holds C_n in the opposite slots of each node
enum { VIEW_DIRECT = 0, VIEW_PULL_PENDING = 1, VIEW_AA_NATURAL = 2, VIEW_AA_SWAPPED = 3 };

void launch_collide_inplace(const DevLattice &d, int cur, int side_par, cudaStream_t s);
void launch_pull(const DevLattice &d, int src, int side_par, bool ghosts, cudaStream_t s);
// Kernels launch_pull launches (16-bit storage without the ghost ring: the quad kernel and the
// perimeter kernel).
int pull_launches(const DevLattice &d, bool ghosts);
void launch_stream(const DevLattice &d, int src, int side_par, cudaStream_t s);
// Pull steps per launch of the tile kernel (tile.cu) for a run of `steps` steps from form C pending:
// 0 where single steps are the faster way (or the only one).  `outlet`: the outlet is
// extrapolated before every step; `rs`: stored values are rounded stochastically.
int tile_steps(const DevLattice &d, long long steps, bool outlet, bool rs);
// T pull steps (a count that tile_steps returned) in one launch: C_n in buffer src (n_par = n & 1)
// -> C_{n+T} in buffer 1 - src, where T single steps would have left it in src: the caller turns
// ghost_flip over and changes the side store's slots' roles (Lattice::after_tile).  keys: rounding keys of the T collisions (16-bit).
void launch_tile(const DevLattice &d, int src, int n_par, int T, bool outlet, const unsigned *keys, cudaStream_t s);
void launch_side_from_buf(const DevLattice &d, int b, int side_par, cudaStream_t s);
// AA only: keep buffer b's ghost ring as the second buffer's (d.ghost2).
void launch_ghost_copy(const DevLattice &d, int b, cudaStream_t s);
void launch_readout(const DevLattice &d, int view, int cur, int side_par, int X0, int X1,
                    double *out, int rec_stride, const uint64_t *dynp, cudaStream_t s);
// launch_readout of a collided pull state as it is (out0) and as its stream gives it (out1; side_par: the
// parity of the collision before).
void launch_readout_both(const DevLattice &d, int cur, int side_par, int X0, int X1, double *out0, double *out1,
                         int rec_stride, const uint64_t *dynp, cudaStream_t s);
// Records of columns X0..X1-1, rows Y0..Y0+H-1 (in: [X - X0][Y - Y0][rec_stride] doubles) into
// buffer b.
void launch_upload(const DevLattice &d, int b, const double *in, int rec_stride, int X0, int X1,
                   int Y0, int H, cudaStream_t s);
// Tag plane from a device copy of a host-order tag array tag_xy[X * (ly + 2) + Y].
void launch_tags_from_xy(const DevLattice &d, const uint8_t *in, cudaStream_t s);
// The extrapolated outlet of the state entering a step: zrho of every row and the tables' slots.
void launch_zgb(const DevLattice &d, int view, int cur, int side_par, cudaStream_t s);
void launch_periodic(const DevLattice &d, int b, cudaStream_t s);
// Tag plane of the cylinder channel (obstacle disk, walls of wall_kind, regularized inlet,
// pressure-regularized outlet) written on the device.
void launch_cylinder_tags(const DevLattice &d, int ox, int oy, int r, int wall_kind, cudaStream_t s);
void launch_init_cylinder(const DevLattice &d, int b, double umax, cudaStream_t s);
// Density and velocity of rows Y0..Y1-1 ([Y - Y0][X - 1]; any pointer may be null).
void launch_macros(const DevLattice &d, int view, int cur, int side_par, int Y0, int Y1, double *rho, double *ux,
                   double *uy, cudaStream_t s);
// out[k] = in[k] * scale
void launch_scaled(const double *in, double scale, double *out, long long n, cudaStream_t s);
// FP64 reductions of the current state (mass, momentum, obstacle force, kinetic energy,
// non-finite nodes, fluid mass) into out[8]; `partial` is scratch of (ly+2)*8 doubles.
void launch_moments(const DevLattice &d, int view, int cur, int side_par, double *partial,
                    double *out, cudaStream_t s);
// acc[0..lx*ly) += ux, acc[lx*ly..2*lx*ly) += uy of the current state.
void launch_accumulate_velocity(const DevLattice &d, int view, int cur, int side_par, double *acc,
                                cudaStream_t s);
// max over the interior of |u - u_prev| into *out (float bits, cleared by the caller);
// prev (lx*ly float2, [Y-1][X-1]) receives the current velocity.
void launch_velocity_change(const DevLattice &d, int view, int cur, int side_par, void *prev,
                            unsigned *out, cudaStream_t s);
// ---- batches: many lattices per launch ------------------------------------------------
// threads per block = nodes per tile: 128, 256 or 512
// Kinds of batch step: pull (one node per thread), AA even and odd, the 16-bit pull with four
// nodes per thread (each warp one row of 128 nodes, see pull_quad), which leaves each member's
// perimeter nodes to BATCH_PERIM: the pull step of those nodes, one per thread, one block a run
// of `threads` perimeter nodes of a member (work item: the member, x0 = the run's first number).
enum { BATCH_PULL = 0, BATCH_AA_EVEN = 1, BATCH_AA_ODD = 2, BATCH_PULL4 = 3, BATCH_PERIM = 4 };
constexpr int BATCH_KINDS = 5;

// One lattice of a batch, with its state at the start of the current chunk of steps:
// pull scheme: the buffer holding C_n is buf[cur0]; AA: phase0 0 = natural form, 1 = swapped;
// tau0 = the time step the chunk's first launch executes (its side parity is tau0 & 1).
// What every block reads lies in one 128-byte line (a second line: AA members of 1500 x 400 in FP32 124.7 us a step, 119.9
// without it).
struct alignas(128) BatchInst {
    Geo g;
    void *buf[2];
    void *side;
    const uint8_t *tag;
    const double *bc;
    double omega;
    float scale, inv_scale;
    int tau0;                         // tau0 + k: the collision number of step k of a chunk
    int cur0;
    int side_slot;                    // of each collision parity (batch_side_slot)
    int rules_inside;
    int scheme, phase0;
    unsigned rs_seed;                 // 16-bit members: stochastic rounding seed (rs != 0)
    int rs;
};
static_assert(sizeof(Geo) == 56 && sizeof(BatchInst) == 256, "the first line holds all up to rules_inside");

// One word for both parities' slots: with a pointer for each the kernels keep what they can otherwise compute again, and
// spill (FP16 pull, 32 registers: 104 bytes instead of 8; 64 channels of 100 x 60 with row-shifted offsets 25.9
// us a step on one B200 instead of 22.9, AA ones in FP32 16.8 and 15.7).
__host__ __device__ inline int batch_side_slot(int slots, int parity) { return (slots >> (8 * parity)) & 0xff; }
__host__ __device__ inline int batch_side_slots(int even, int odd) { return even | (odd << 8); }

// A strip of `passes` tiles of a lattice stacked in y, stepped by one block from the top down.
// A tile: nodes x0 .. x0 + (32 << shape) - 1 and threads / (32 << shape) rows (BATCH_PULL4:
// x0 .. x0 + 127 and threads / 32 rows); pass p covers the tile starting at row
// y0 + p * (rows of a tile).  `sp` packs shape (bits 0..7) and passes (bits 8..).
struct BatchWork {
    int inst, x0, y0, sp;
};
__host__ __device__ inline int batch_shape(int sp) { return sp & 0xff; }
__host__ __device__ inline int batch_passes(int sp) { return sp >> 8; }
__host__ __device__ inline int batch_sp(int shape, int passes) { return shape | (passes << 8); }

// Step k of a chunk, of kind BATCH_PULL / AA_EVEN / AA_ODD / PULL4 (16-bit only), for every tile of a
// work list of `nwork` tiles of `threads` nodes: `persistent` grids of `grid` blocks stride
// through the list, otherwise `grid` must equal nwork (one block per tile).
// flags (16-bit batches): bit 0 -- some member rounds stochastically, bit 1 -- some member stores
// row-shifted offsets; the kernels then carry those paths.
void launch_batch(int precision, int kind, int threads, bool persistent, int flags, const BatchInst *insts,
                  const BatchWork *work, int nwork, int grid, int k, cudaStream_t s);
// The batch's tile kernel (tile.cu): nodes of a tile; and two steps (BATCH_TILE_STEPS) of every tile of a work
// list, launch `unit` since the descriptors (rs: some member rounds stochastically).
constexpr int BATCH_TILE_STEPS = 2;
void batch_tile(int precision, int *w, int *h);
void launch_batch_tile(int precision, bool rs, const BatchInst *insts, const BatchWork *work, int nwork, int unit, cudaStream_t s);
// Resident blocks per SM of the persistent kernel of a kind and block size.
int batch_blocks_per_sm(int precision, int kind, int threads);

// AA scheme (buffer 0): the even step collides every node in place into the opposite slots,
// the odd step gathers from the neighbours' opposite slots and scatters to their natural slots.
void launch_aa_even(const DevLattice &d, int side_par, cudaStream_t s);
void launch_aa_odd(const DevLattice &d, int side_par, cudaStream_t s);

}  // namespace lbgpu
