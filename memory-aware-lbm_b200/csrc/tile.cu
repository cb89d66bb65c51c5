// tile.cu -- runs of pull steps, several steps a launch on tiles in shared memory (tile.cuh): which
// shape of tile a lattice takes, and the launch.
#include "kernels.h"
#include "node.cuh"

namespace lbgpu {

namespace {

#include "tile.cuh"

// The shapes by storage type and node count, from a sweep of about ten shapes over channels of 250 x 51 to 8192 x
// 2048 (us a step in a graph of launches; the next best shape or the single-step kernel in parentheses):
//   small lattices: many steps a launch on small tiles, so that every SM has a tile and the launch is
//     shared: FP64 250 x 51 2.4 (4 steps 2.8, single 3.5), FP32 1.5 (1.9, 3.3), FP16 2.0 (2.2, 6.7)
//     (to 19K nodes, a tile a SM; FP16 1.8 on 704 threads); 400 x 90: FP64 3.1 with 4 steps (4.0 with 8), FP32
//     2.1 with two tiles a SM (2.5 with one), FP16 2.2 (2.6)
//   511 x 127: FP64 3.8 (5.0 with 2 steps, single 4.0), FP32 2.5 (2.6 with 8 steps, single 3.5)
//   700 x 200: FP64 5.4 (5.6 with 2 steps), FP32 2.9 (3.2 on 32 x 8 tiles, single 4.3), FP16 3.4 (3.5 on 416 threads, single 7.2)
//   1024 x 256: FP64 7.4 (8.3 with 4 steps, single 7.0 in a graph and 9.0 launched), FP32 4.2 (5.2 with 2, 5.5)
//   2047 x 511: FP64 21.9 (24.2 on 64 x 16, single 27.7), FP32 10.1 (11.1 with 4 steps, 12.8), FP16 8.9 (10.0 with 2 steps, 12.3)
//   large: two steps, tiles whose halo is small against them, and few enough threads' registers for
//     several blocks a SM: 8192 x 2048 FP64 233 (two blocks of 64 x 16; 236 with four of 32 x 16; single 355), FP32
//     109 (five of 64 x 12; 111 with six of 64 x 8; single 187), FP16 93 (97 with prefetch; single 109);
//     16384 x 4096 FP16 342 (single 388), with stochastic rounding 398 (single 398: its hash and
//     multiplies bind), so those keep k_pull4h from 24M nodes on; 4096 x 1024 31 and 38.  Row-shifted FP16 110 (single
//     117) at 8192 x 2048, 420 (408) at 16384 x 4096: from 24M nodes too; both together 34.9 (39.4) at 4096 x 1024,
//     126 (117) at 8192 x 2048, 65.6 (62.4) at 6926 x 1153, 43.3 (41.5) at 7745 x 645, 40.8 (42.8) at 5438 x 906: from 4.7M.
// Large lattices prefetch the tile 100 (FP64) or 200 (FP32) blocks ahead into L2: 253 -> 233 and 120 -> 109 us;
// 0.3 of that distance does half as much, 4 times it costs 15-30 % (evicted before it is read).
using F64Small = TileShape<double, 16, 8, 8, 704, 1>;
using F64Mid = TileShape<double, 32, 8, 4, 288, 2>;
using F64Wide = TileShape<double, 32, 8, 2, 352, 3>;
using F64Large = TileShape<double, 64, 16, 2, 512, 2>;
using F32Small = TileShape<float, 16, 8, 8, 768, 1>;
using F32Small2 = TileShape<float, 16, 8, 8, 384, 2>;
using F32Mid = TileShape<float, 32, 8, 4, 288, 3>;
using F32Wide = TileShape<float, 32, 16, 4, 448, 2>;
using F32Large = TileShape<float, 64, 12, 2, 224, 5>;
// Batches advance every member by the same steps, two at a time, and fill the GPU: the large lattices' tiles,
// with FP64's in halves because members are small (71 against 72 GLUPS on one large lattice).
using F64Batch = TileShape<double, 32, 16, 2, 256, 4>;
using F32Batch = F32Large;
template <class S> using HalfSmall = TileShape<S, 16, 8, 8, 704, 1>;
template <class S> using HalfSmall2 = TileShape<S, 16, 8, 8, 384, 2>;
template <class S> using HalfWide = TileShape<S, 32, 16, 4, 448, 3>;
template <class S> using HalfLarge = TileShape<S, 64, 12, 2, 224, 5>;

enum { TILE_SMALL = 0, TILE_MID = 1, TILE_WIDE = 2, TILE_LARGE = 3, TILE_NONE = 4 };

// Node counts below which a shape is the fastest.
constexpr long long kF64[3] = {19 << 10, 120 << 10, 3 << 20};
constexpr long long kF32[3] = {52 << 10, 100 << 10, 700 << 10};
constexpr long long kHalf[3] = {60 << 10, 60 << 10, 2 << 20};
bool elem16(const DevLattice &d) { return d.precision == LBGPU_F16 || d.precision == LBGPU_BF16; }

// Up to here the small tiles (128 nodes) are one a SM, and take all its threads; beyond, two share one.
constexpr long long kOneASm = 148 * 128;

// Lattices that are only some tiles high or wide are nearly all halo and edge (us a step, single steps in parentheses):
//   FP64 large tiles, 64 x 16: 250000 x 20 130 (122), 66 x 65000 211 (197), against 120 and 201 on 32 x 8 tiles, which
//     are ahead up to 256 rows or columns, but for 12 to 16 rows; 33 to 64 columns are one tile of 64 x 16, ahead from
//     600K nodes on: 33 x 20000 44 and 53 (51).
//   16-bit tiles of 32 x 16, four steps, up to 35 rows (none of them off the perimeter): 250000 x 5 29 (27), 60000 x 32 22.3
//     (19.6), against 22.6 and 18.0 on 64 x 12; the line lies where both run alike.
//   Row-shifted offsets, whose four steps spill registers: 64 x 12 tiles are ahead from 600K nodes (1937 x 968 22.0 and
//     15.4, single 21.3).
int tile_shape(const DevLattice &d, bool rs)
{
    const int lx = d.g.lx, ly = d.g.ly;
    const long long n = (long long)lx * ly;
    const long long *k = d.precision == LBGPU_F64 ? kF64 : (d.precision == LBGPU_F32 ? kF32 : kHalf);
    const int shape = n < k[0] ? TILE_SMALL : (n < k[1] ? TILE_MID : (n < k[2] ? TILE_WIDE : TILE_LARGE));
    if (d.precision == LBGPU_F64 && shape >= TILE_WIDE) {
        if (lx > 32 && lx <= 64) return n >= (600ll << 10) ? TILE_LARGE : TILE_WIDE;
        if ((ly < 256 && (ly < 12 || ly > 16)) || lx < 256) return TILE_WIDE;
    }
    if (shape == TILE_WIDE && elem16(d) &&
        n >= (d.g.shift_u ? 600ll << 10 : (ly <= 35 ? (rs ? 700ll << 10 : 1ll << 20) : kHalf[2])))
        return TILE_LARGE;
    return shape;
}

// Lattices whose single steps are the faster way for their shape (the same sweeps): a few long rows, whose nodes are
// nearly all computed in tiles of edges, while a single step streams them well.  `rules`: where the first and
// last row are boundary rules, which every tile then lists.
struct Flat {
    int rows, to;              // rows of the lattice
    long long nodes, below;    // its nodes
    int ratio;                 // nodes a row for each row, at least
    bool rules;
};
constexpr long long kK = 1 << 10, kM = 1 << 20, kAny = 1ll << 62;
// FP64 60000 x 10 22.3 (16.4), 1000000 x 3 142 (97); 12 to 14 rows fill a tile of 64 x 16: 1000000 x 12 278 (291).  Rules: 250000 x
// 20 189 (136), 8000 x 16 9.3 (6.5).
constexpr Flat kFlat64[] = {{1, 11, 170 * kK, kAny, 0, false}, {12, 14, 170 * kK, 3 * kM, 0, false}, {15, 16, 900 * kK, kAny, 0, false},
                            {1, 48, 170 * kK, kAny, 0, true}, {1, 48, 100 * kK, kAny, 300, true}};
// FP32 60000 x 3 8.7 (6.2), 1000000 x 5 90 (76).  Rules: 60000 x 10 15.4 (10.5), 20000 x 32 12.3 (10.3), 1000000 x 16 263 (241).
constexpr Flat kFlat32[] = {{1, 8, 170 * kK, kAny, 0, false}, {1, 32, 150 * kK, 1300 * kK, 500, true},
                            {1, 20, 1300 * kK, 2 * kM, 500, true}, {1, 16, 2 * kM, kAny, 500, true}};
// 16-bit: two rows of tiles of 64 x 12, none off the perimeter: 1000000 x 16 184 (152).  Rules: 250000 x 3 43.5 (28.7), 1000000 x
// 32 320 (282).
constexpr Flat kFlat16[] = {{13, 25, 1 * kM, kAny, 0, false}, {1, 12, 500 * kK, kAny, 0, true}, {26, 35, 4 * kM, kAny, 0, true}};
// with stochastic rounding 60000 x 24 23 (16.7), 1000000 x 8 118 (108).  Rules: 60000 x 5 13.9 (12.3), 250000 x 48 124 (112).
constexpr Flat kFlat16R[] = {{13, 35, 700 * kK, kAny, 0, false}, {1, 12, 6 * kM, kAny, 0, false}, {1, 12, 290 * kK, kAny, 0, true},
                             {1, 56, 6 * kM, kAny, 0, true}};
// with a row shift 60000 x 24 30.6 (14.9), 20000 x 20 11.2 (8.2); from 64 rows on both run alike.  Rules: 60000 x 64 37.9 (34.9).
constexpr Flat kFlat16B[] = {{1, 63, 250 * kK, kAny, 64, false}, {1, 63, 58 * kK, kAny, 256, false}, {64, 100, 3 * kM, kAny, 64, true}};
// with both 60000 x 96 54 (47), 20000 x 32 15.4 (10.2).
constexpr Flat kFlat16BR[] = {{1, 1 << 30, 250 * kK, kAny, 64, false}, {1, 1 << 30, 58 * kK, kAny, 128, false}};

template <size_t N>
bool on_lines(const Flat (&lines)[N], const DevLattice &d, bool outlet)
{
    const long long n = (long long)d.g.lx * d.g.ly;
    for (const Flat &f : lines)
        if (d.g.ly >= f.rows && d.g.ly <= f.to && n >= f.nodes && n < f.below && d.g.lx >= (long long)f.ratio * d.g.ly &&
            (d.row_rules || !f.rules) &&
            // the pass of an extrapolated outlet makes a single step longer, but for FP64's rules
            (!outlet || n >= kM || (f.rules && d.precision == LBGPU_F64)))
            return true;
    return false;
}

bool too_flat(const DevLattice &d, bool outlet, bool rs)
{
    if (d.precision == LBGPU_F64)      // and narrow ones: 66 x 65000 201 (197)
        return on_lines(kFlat64, d, outlet) || (d.g.lx > 64 && d.g.lx <= 100 && (long long)d.g.lx * d.g.ly >= 4 * kM);
    if (d.precision == LBGPU_F32) return on_lines(kFlat32, d, outlet);
    if (d.g.shift_u) return rs ? on_lines(kFlat16BR, d, outlet) : on_lines(kFlat16B, d, outlet);
    return rs ? on_lines(kFlat16R, d, outlet) : on_lines(kFlat16, d, outlet);
}

template <class SH, int M, bool EXTRAP>
void launch_shape(const DevLattice &d, int src, int n_par, int pf, const unsigned *keys, cudaStream_t s)
{
    using S = typename SH::S;
    TileArgs<S> a;
    a.g = d.g;
    a.src = B<S>(d, src);
    a.dst = B<S>(d, 1 - src);
    a.tag = d.tag;
    a.bc = d.bc;
    a.zgb = d.zgb_src + 3 * d.g.nb;
    a.omega = d.omega;
    a.omega_f = (float)d.omega;
    // step 1 reads the stale slots of C_{n-1}; the last step's replace those of C_n, which has them in
    // its own slots, and the step's before it go to a free slot.  Row-shifted offsets read C_n's from
    // the side store too (its own slots are rebased), so both go to free slots, of four.
    a.stale1 = SIDE<S>(d, n_par + 1);
    a.stale2 = SIDE<S>(d, n_par);
    a.out_last = (M & TILE_SHIFT) ? SIDE_SLOT<S>(d, side_other(d, n_par)) : SIDE<S>(d, n_par);
    a.out_prev = SIDE_SLOT<S>(d, side_other(d, 1 - n_par));
    a.sc = d.scale;
    a.inv = d.inv_scale;
    // the outlet's extrapolation reads three columns back: its tile must not be narrower
    a.x_first = EXTRAP && d.g.lx > SH::W && (d.g.lx % SH::W == 1 || d.g.lx % SH::W == 2) ? -3 : 1;
    a.nx = (int)cdiv(d.g.lx - a.x_first + 1, SH::W);
    a.ny = (int)cdiv(d.g.ly, SH::H);
    // a long launch loses more to the ring's rows read out of order than its tail costs (FP32 16384 x 4096 414 us a
    // step row by row, 433 ring first; 4096 x 1024 35.5 and 34.0, 1024 x 256 4.8 and 3.6; FP64 is faster ring first throughout)
    a.ring_first = sizeof(S) == 8 || (long long)a.nx * a.ny < 12000;
    a.pf = a.x_first == 1 ? pf : 0;
    a.rules_inside = d.rules_inside;
    for (int k = 0; k < 8; ++k) a.keys[k] = keys[k];
    cudaFuncSetAttribute(k_tile<SH, M, EXTRAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::SMEM);
    k_tile<SH, M, EXTRAP><<<(unsigned)a.nx * (unsigned)a.ny, SH::NT, SH::SMEM, s>>>(a);
}

template <class SH>
void launch_one(const DevLattice &d, int src, int n_par, bool outlet, int pf, const unsigned *keys, cudaStream_t s)
{
    if constexpr (sizeof(typename SH::S) == 2) {
        if constexpr (SH::T < 8) {
            if (d.g.shift_u) {
                if (keys[0] != 0) launch_shape<SH, TILE_RS | TILE_SHIFT, false>(d, src, n_par, pf, keys, s);
                else launch_shape<SH, TILE_SHIFT, false>(d, src, n_par, pf, keys, s);
                return;
            }
        }
        if (keys[0] != 0) {
            if (outlet) launch_shape<SH, TILE_RS, true>(d, src, n_par, pf, keys, s);
            else launch_shape<SH, TILE_RS, false>(d, src, n_par, pf, keys, s);
            return;
        }
    }
    if (outlet) launch_shape<SH, 0, true>(d, src, n_par, pf, keys, s);
    else launch_shape<SH, 0, false>(d, src, n_par, pf, keys, s);
}

template <class S>
void launch_half(const DevLattice &d, int src, int n_par, int T, bool outlet, const unsigned *keys, cudaStream_t s)
{
    if (T == 8 && (long long)d.g.lx * d.g.ly <= kOneASm) launch_one<HalfSmall<S>>(d, src, n_par, outlet, 0, keys, s);
    else if (T == 8) launch_one<HalfSmall2<S>>(d, src, n_par, outlet, 0, keys, s);
    else if (T == 4) launch_one<HalfWide<S>>(d, src, n_par, outlet, 0, keys, s);
    else launch_one<HalfLarge<S>>(d, src, n_par, outlet, 0, keys, s);
}

}  // namespace

int tile_steps(const DevLattice &d, long long steps, bool outlet, bool rs)
{
    if (steps < 2 || (outlet && !d.outlet_tiles) || too_flat(d, outlet, rs)) return 0;
    const int shape = tile_shape(d, rs);
    const long long nodes = (long long)d.g.lx * d.g.ly;
    // A rest of two or three steps on a small lattice, whose tiles of two steps are too few and too large for the GPU: a
    // launch of two and two single steps, FP32 250 x 51 11.4 and 10.3 us, row-shifted 400 x 90 15.8 and 12.4.
    if (steps < 4 && !outlet && ((d.precision == LBGPU_F32 && nodes < (30ll << 10)) || (d.g.shift_u && nodes < (100ll << 10)))) return 0;
    if (elem16(d)) {
        if (d.g.shift_u && outlet) return 0;
        if (nodes >= (rs && d.g.shift_u ? 9ll << 19 : 24ll << 20) && (rs || d.g.shift_u)) return 0;
        return shape == TILE_SMALL && steps >= 8 && !d.g.shift_u ? 8 : (steps >= 4 && shape != TILE_LARGE ? 4 : 2);
    }
    if (shape == TILE_SMALL && steps >= 8) return 8;
    if (steps >= 4 && (shape <= TILE_MID || (shape == TILE_WIDE && d.precision == LBGPU_F32))) return 4;
    return 2;
}

void launch_tile(const DevLattice &d, int src, int n_par, int T, bool outlet, const unsigned *keys, cudaStream_t s)
{
    const int shape = tile_shape(d, keys[0] != 0);
    switch (d.precision) {
    case LBGPU_F64:
        if (T == 8) launch_one<F64Small>(d, src, n_par, outlet, 0, keys, s);
        else if (T == 4) launch_one<F64Mid>(d, src, n_par, outlet, 0, keys, s);
        else if (shape == TILE_LARGE) launch_one<F64Large>(d, src, n_par, outlet, 100, keys, s);
        else launch_one<F64Wide>(d, src, n_par, outlet, 0, keys, s);
        break;
    case LBGPU_F32:
        if (T == 8 && (long long)d.g.lx * d.g.ly <= kOneASm) launch_one<F32Small>(d, src, n_par, outlet, 0, keys, s);
        else if (T == 8) launch_one<F32Small2>(d, src, n_par, outlet, 0, keys, s);
        else if (T == 4 && shape == TILE_WIDE) launch_one<F32Wide>(d, src, n_par, outlet, 0, keys, s);
        else if (T == 4) launch_one<F32Mid>(d, src, n_par, outlet, 0, keys, s);
        else launch_one<F32Large>(d, src, n_par, outlet, shape == TILE_LARGE ? 200 : 0, keys, s);
        break;
    case LBGPU_F16: launch_half<__half>(d, src, n_par, T, outlet, keys, s); break;
    default: launch_half<__nv_bfloat16>(d, src, n_par, T, outlet, keys, s); break;
    }
}

namespace {

template <class SH, bool RS>
void launch_batch_shape(const BatchInst *insts, const BatchWork *work, int nwork, int unit, cudaStream_t s)
{
    cudaFuncSetAttribute(k_batch_tile<SH, RS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::SMEM);
    k_batch_tile<SH, RS><<<nwork, SH::NT, SH::SMEM, s>>>(insts, work, unit);
}

template <class S>
void launch_batch_half(bool rs, const BatchInst *insts, const BatchWork *work, int nwork, int unit, cudaStream_t s)
{
    if (rs) launch_batch_shape<HalfLarge<S>, true>(insts, work, nwork, unit, s);
    else launch_batch_shape<HalfLarge<S>, false>(insts, work, nwork, unit, s);
}

}  // namespace

void batch_tile(int precision, int *w, int *h)
{
    *w = precision == LBGPU_F64 ? F64Batch::W : (precision == LBGPU_F32 ? F32Batch::W : HalfLarge<__half>::W);
    *h = precision == LBGPU_F64 ? F64Batch::H : (precision == LBGPU_F32 ? F32Batch::H : HalfLarge<__half>::H);
}

void launch_batch_tile(int precision, bool rs, const BatchInst *insts, const BatchWork *work, int nwork, int unit,
                       cudaStream_t s)
{
    switch (precision) {
    case LBGPU_F64: launch_batch_shape<F64Batch, false>(insts, work, nwork, unit, s); break;
    case LBGPU_F32: launch_batch_shape<F32Batch, false>(insts, work, nwork, unit, s); break;
    case LBGPU_F16: launch_batch_half<__half>(rs, insts, work, nwork, unit, s); break;
    default: launch_batch_half<__nv_bfloat16>(rs, insts, work, nwork, unit, s); break;
    }
}

}  // namespace lbgpu
