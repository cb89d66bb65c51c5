// tile.cuh -- several pull steps per launch on tiles held in shared memory (k_tile).
//
// Included by tile.cu inside its namespace: it uses the per-node functions of node.cuh, so a node's
// result is the same bits as in a single-step kernel.
//
// A block advances a tile of W x H nodes T steps.  Step s computes the tile and a halo of T - s nodes
// around it (what the tile's last step needs of its neighbours, computed again by each of them):
// step 1 gathers C_n from the planes, the steps between live in one or two shared buffers, step T
// writes C_{n+T} to the other buffer's planes.  So the lattice crosses the memory once per T steps
// and a launch is paid once per T steps; no block waits for another.
//
// What it measured (one B200, channel lattices, us a step, single-step kernel -> tiles, both as
// lbgpu_step runs them):
//   FP64  250 x 51     6.2 -> 2.6   (launch rate -> the boundary rules' chain of dependent operations)
//   FP64  16384 x 4096 1476 -> 978  (HBM -> 68 GLUPS at 67 B an update, FP64 pipe half busy)
//   FP32  1024 x 256   8.2 -> 3.6
//   FP32  8192 x 2048  189 -> 111   (HBM -> 151 GLUPS at 32 B an update, 114 instructions an update)
//   FP16  2047 x 511   14.4 -> 7.7, 4096 x 1024 36 -> 26, 16384 x 4096 384 -> 346 (issue: 139 instructions an update in
//         k_pull4h), with stochastic rounding 14.9 -> 9.3, 37.8 -> 29.7 (the single kernel from 24M nodes on)
// Loading the tiles by TMA instead (whole boxes of nine planes into a third buffer, results stored by TMA)
// ran at 124-129 GLUPS where this form had 134 (FP32 before the pairs) and 63 against 67 (FP64): the extra
// buffer costs resident blocks, and their overlap is what hides the latencies of both halves.
#pragma once

// Shape of a tile kernel: W x H nodes advanced T steps by NT threads, MINB blocks a SM.  Step 1's region is RW x RH;
// two buffers of that size alternate between the steps (one where T is 2).
template <class S_, int W_, int H_, int T_, int NT_, int MINB_>
struct TileShape {
    using S = S_;
    static constexpr int W = W_, H = H_, T = T_, NT = NT_, MINB = MINB_;
    static constexpr int RW = W + 2 * (T - 1), RH = H + 2 * (T - 1);   // region of step 1
    static constexpr int PL = RW * RH;                                 // elements a plane of a buffer
    static constexpr int NBUF = T > 2 ? 2 : 1;
    static constexpr int TAGS = (PL + 15) / 16 * 16;                   // bytes of the tag copy
    // buffer 1 starts one element later, so that the pairs that each step stores lie on pair boundaries
    static constexpr size_t B1 = 9 * (size_t)PL + 1;                   // element of buffer 1
    static constexpr size_t POPS = (((NBUF == 2 ? B1 + 1 : 0) + 9 * (size_t)PL) * sizeof(S) + 15) / 16 * 16;
    static constexpr size_t LIST = POPS + TAGS;
    static constexpr size_t SMEM = LIST + (2 * (size_t)PL + 15) / 16 * 16 + 16;
    static_assert(W % 2 == 0 && T % 2 == 0, "pairs of nodes");
};

// Modes of 16-bit storage (M): stochastic rounding, row-shifted offsets.
enum { TILE_RS = 1, TILE_SHIFT = 2 };

template <class S>
struct TileArgs {
    Geo g;
    const S *src;
    S *dst;
    const uint8_t *tag;
    const double *bc;
    const int *zgb;            // [nb] of the right pressure table: >= 0 where the outlet is extrapolated
    double omega;
    const S *stale1;           // stale slots of C_{n-1}, read by step 1
    const S *stale2;           // and of C_n, by step 2 (row-shifted offsets: the planes' are rebased)
    S *out_last, *out_prev;    // where the stale slots of C_{n+T} and C_{n+T-1} go
    float sc, inv, omega_f;
    int x_first;               // column of the first tile (1, or less, see launch_tile)
    int nx, ny;                // tiles
    int ring_first;            // their order (tile_place)
    int pf;                    // tiles ahead whose nodes are prefetched into L2
    int rules_inside;          // some node off the perimeter has a boundary rule
    unsigned keys[8];          // stochastic rounding keys of the steps
};

// Block b's tile: row by row, or the outer ring of tiles first (their boundary rules make them the longest, and
// a launch ends with its last block) and then the others row by row.
__device__ __forceinline__ void tile_place(unsigned b, int nx, int ny, int ring_first, int &tx, int &ty)
{
    if (!ring_first || nx < 3 || ny < 3) {
        ty = (int)(b / (unsigned)nx);
        tx = (int)(b - (unsigned)ty * (unsigned)nx);
        return;
    }
    const unsigned ring = 2u * (unsigned)(nx + ny) - 4u;
    if (b >= ring) {
        const unsigned k = b - ring, r = k / (unsigned)(nx - 2);
        ty = 1 + (int)r;
        tx = 1 + (int)(k - r * (unsigned)(nx - 2));
        return;
    }
    const int k = (int)b;
    if (k < nx) { tx = k; ty = 0; }
    else if (k < 2 * nx) { tx = k - nx; ty = ny - 1; }
    else { tx = (k - 2 * nx) & 1 ? nx - 1 : 0; ty = 1 + (k - 2 * nx) / 2; }
}

// The slots of perimeter node (X, Y) that no interior node streams into: F(i) for each.
template <class FN>
__device__ __forceinline__ void stale_slots(const Geo &g, int X, int Y, FN fn)
{
    const bool l = X == 1, r = X == g.lx, b = Y == 1, t = Y == g.ly;
    if (l) fn(1);
    if (b) fn(2);
    if (r) fn(3);
    if (t) fn(4);
    if (l || b) fn(5);
    if (r || b) fn(6);
    if (r || t) fn(7);
    if (l || t) fn(8);
}

// Stores a collided node of step s, and keeps the stale slots of a perimeter node (those no interior
// node streams into hold the node's own value of two steps before): each lies in the ghost cell
// that a gather reads for it, which no other node reads or writes, in the buffer that step s + 2
// reads; after the last two steps they also go to the side store.
template <class S, class SH, int s, bool EDGE, int M>
__device__ __forceinline__ void tile_store(const TileArgs<S> &a, const typename Work<S>::W f[9], S *__restrict__ rd,
                                           S *__restrict__ wr, S *const gd[9], unsigned go, int X, int Y, int q, bool owned)
{
    const Geo &g = a.g;
    constexpr int RW = SH::RW, PL = SH::PL;
    constexpr bool RS = (M & TILE_RS) != 0, SHIFT = (M & TILE_SHIFT) != 0;
    const RsNode h = rs_node<S, RS>(g, a.keys[s - 1], X, Y);
    S v[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = put<S, RS>(stored_out<S, SHIFT ? 1 : 0>(g, Y, i, f[i], a.sc), i, a.sc, h);
    if (s == SH::T) {
#pragma unroll
        for (int i = 0; i < 9; ++i) *reinterpret_cast<S *>(reinterpret_cast<char *>(gd[i]) + go) = v[i];
    } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) wr[i * PL + q] = v[i];
    }
    if (EDGE && g.perimeter(X, Y)) {
        const int p = g.pidx(X, Y);
        const int c = q % RW, r = q / RW;
        stale_slots(g, X, Y, [&](int i) {
            const int dx = (i == 1 || i == 5 || i == 8) ? 1 : ((i == 3 || i == 6 || i == 7) ? -1 : 0);
            const int dy = (i == 2 || i == 5 || i == 6) ? 1 : ((i == 4 || i == 7 || i == 8) ? -1 : 0);
            S w = v[0];                 // (relative to the node's own row: it is the one that reads it)
#pragma unroll
            for (int j = 1; j < 9; ++j) if (i == j) w = SHIFT ? put<S, RS>(f[j], j, a.sc, h) : v[j];
            const bool in = c - dx >= 0 && c - dx < RW && r - dy >= 0 && r - dy < SH::RH;
            // the ghost cell that feeds this slot at step s + 2
            if (s + 2 <= SH::T && in) rd[i * PL + q - dy * RW - dx] = w;
            // and at step 2, which reads C_n
            if (s == 1 && in) wr[i * PL + q - dy * RW - dx] =
                SHIFT ? a.stale2[(size_t)i * g.nper + p] : a.src[(size_t)i * (size_t)g.plane + g.idx(X, Y)];
            if (s == SH::T) a.out_last[(size_t)i * g.nper + p] = w;
            if (s == SH::T - 1 && owned) a.out_prev[(size_t)i * g.nper + p] = w;
        });
    }
}

// Density of the state entering step s at column lx - 1 - j of row Y (the extrapolated outlet).
template <class S, class SH, int s>
__device__ __forceinline__ double tile_density(const TileArgs<S> &a, const S *__restrict__ rd, int X, int Y, int q, int j)
{
    using R = typename Codec<S>::R;
    const Geo &g = a.g;
    const int Xj = g.lx - 1 - j, qj = q + (Xj - X);
    const long long oj = g.idx(Xj, Y);
    R h[9];
#pragma unroll
    for (int i = 0; i < 9; ++i)
        h[i] = dec_row<S>(g, s == 1 ? plane(a.src, g, i)[oj - cx(i) - (long long)cy(i) * g.pitch]
                                    : rd[i * SH::PL + qj - cy(i) * SH::RW - cx(i)], i, a.inv, Y);
    return (double)rules::density(h);
}

// A boundary rule in exact FP64, out of line.  Tiles of 64 columns go through the general dispatch, whose BGK no rule takes:
// with it the compiler spills less around the call (64 x 16, 8192 x 2048 with the extrapolated outlet 254 us a step on
// one B200 and 276 without it, 16384 x 4096 982 and 1004); smaller ones are faster without (250 x 51 2.65 and 2.78).
template <class SH>
__device__ __forceinline__ void tile_rule(int t, double f[9], double omega, double p0, double p1)
{
    if constexpr (SH::W >= 64) rules::collide<double, true>(t, f, omega, p0, p1);
    else rules::collide_called<double, true>(t, f, omega, p0, p1);
}

// The boundary rules (tags of 3 and more) at one node.
template <class S, class SH, int s, int M, bool EXTRAP>
__device__ __forceinline__ void tile_boundary(const TileArgs<S> &a, const S *__restrict__ rd, int t, int X, int Y, int q,
                                              typename Work<S>::W f[9])
{
    const Geo &g = a.g;
    if (EXTRAP && (t == LBGPU_TAG_RIGHT_PRESSURE_ZOUHE || t == LBGPU_TAG_RIGHT_PRESSURE_REGULARIZED) && a.zgb[Y] >= 0) {
        using D = Ar<double>;
        const double r1 = tile_density<S, SH, s>(a, rd, X, Y, q, 0), r2 = tile_density<S, SH, s>(a, rd, X, Y, q, 1);
        const double rho = D::S(D::M(4. / 3., r1), D::M(1. / 3., r2));
        if constexpr (sizeof(S) == 8) tile_rule<SH>(t, f, a.omega, rho, 0.0);
        else collide_given<S>(g, t, f, a.omega, a.sc, a.inv, rho, 0.0);
    } else if constexpr (sizeof(S) == 8 && SH::T == 4) {
        // in line: the call's way through local memory is part of a step's longest chain.  FP64 511 x 127 3.8 -> 3.4
        // us a step; eight steps' copies of it leave the instruction cache (250 x 51 2.4 -> 2.9), and FP32 gains
        // nothing.
        double p0, p1;
        node_params(a.bc, g, t, X, Y, p0, p1);
        rules::boundary_rule<double, true>(t, f, a.omega, p0, p1);
    } else if constexpr (sizeof(S) == 8 && SH::W >= 64) {
        collide_node<S, true>(a.bc, g, t, X, Y, f, a.omega);
    } else if constexpr (sizeof(S) == 8) {
        double p0, p1;
        node_params(a.bc, g, t, X, Y, p0, p1);
        rules::collide_called<double, true>(t, f, a.omega, p0, p1);
    } else {
        collide_w<S, (M & TILE_SHIFT) ? 1 : 0>(a.bc, g, t, X, Y, f, a.omega, a.sc, a.inv);
    }
}

// Bulk, bounce-back and rule-less nodes.
template <class S, int M>
__device__ __forceinline__ void tile_bulk(const TileArgs<S> &a, int t, int X, int Y, typename Work<S>::W f[9])
{
    if constexpr ((M & TILE_SHIFT) != 0) {
        collide_w<S, 1>(a.bc, a.g, t, X, Y, f, a.omega, a.sc, a.inv);
        return;
    }
    if constexpr (sizeof(S) == 2) {
        if (t == TAG_BGK) {
            bgk_offsets<false>(f, a.omega_f, a.sc, a.inv, 0.0f);
            return;
        }
        // boundary_offsets decodes and encodes around its rule
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = (fmaf(f[i], a.inv, wgtf(i)) - wgtf(i)) * a.sc;
    } else {
        if (t == TAG_BGK) {
            if constexpr (sizeof(S) == 8) rules::bgk_exact(f, a.omega);
            else rules::bgk<float>(f, a.omega_f);
            return;
        }
    }
    if (t == TAG_BOUNCE) rules::bounce(f);
}

// Step s (1..T) of the tile: the region of W + 2 (T - s) by H + 2 (T - s) nodes, one node a thread.  Only
// blocks whose region stays off the perimeter (all but FP64 then run tile_step_pairs) have EDGE
// false and skip the tests of lattice bounds.  Nodes with boundary rules (250-500 operations, mostly one after
// another) are listed at step 1 and run packed in warps of their own beside the others: left in
// their places, one or two lanes of every row's warp would hold the whole warp that long.
template <class S, class SH, int s, bool EDGE, int M, bool EXTRAP>
__device__ __forceinline__ void tile_step(const TileArgs<S> &a, S *__restrict__ sm, uint8_t *__restrict__ stag,
                                          unsigned short *__restrict__ list, int *__restrict__ nlist, int x0, int y0)
{
    using Wk = typename Work<S>::W;
    constexpr int E = SH::T - s, WS = SH::W + 2 * E, HS = SH::H + 2 * E, O = s - 1, RW = SH::RW, PL = SH::PL;
    const Geo &g = a.g;
    S *rd = sm + (size_t)(s & 1) * (SH::NBUF - 1) * SH::B1;                // buffer of step s - 1
    S *wr = sm + (size_t)((s - 1) & 1) * (SH::NBUF - 1) * SH::B1;          // buffer of steps s, s - 2
    const int listed = EDGE && s > 1 ? *nlist : 0;
    // node (r, c) of the region; the global planes are addressed by 32-bit offsets from the region's
    // first node, so that the nine bases are uniform over the block
    const long long o0 = (long long)(y0 - E) * g.pitch + (x0 - E + g.xoff - 1);
    const S *gs[9];
    S *gd[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        gs[i] = a.src + ((long long)i * g.plane + o0 - cx(i) - (long long)cy(i) * g.pitch);
        gd[i] = a.dst + ((long long)i * g.plane + o0);
    }
    const uint8_t *gt = a.tag + o0;
    const unsigned pitch = (unsigned)g.pitch * (unsigned)sizeof(S);
    int c = (int)threadIdx.x % WS, r = (int)threadIdx.x / WS;
#pragma unroll 1
    for (; r < HS; c += SH::NT % WS, r += SH::NT / WS, r += c >= WS ? 1 : 0, c -= c >= WS ? WS : 0) {
        const int X = x0 - E + c, Y = y0 - E + r;
        const unsigned go = (unsigned)r * pitch + (unsigned)c * (unsigned)sizeof(S);
        if (EDGE && !g.interior(X, Y)) continue;
        const int q = (r + O) * RW + (c + O);
        int t;
        if (s == 1) {
            t = gt[go / (unsigned)sizeof(S)];
            stag[q] = (uint8_t)t;
        } else {
            t = stag[q];
            if (EDGE && t >= TAG_ZOUHE_FIRST) continue;      // a listed node
        }
        Wk f[9];
        if (s == 1) {
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i] = Work<S>::load(*reinterpret_cast<const S *>(reinterpret_cast<const char *>(gs[i]) + go), i, a.inv);
            if (EDGE && g.perimeter(X, Y)) {
                const int p = g.pidx(X, Y);
#pragma unroll
                for (int i = 0; i < 9; ++i)
                    if (!g.interior(X - cx(i), Y - cy(i))) f[i] = Work<S>::load(a.stale1[(size_t)i * g.nper + p], i, a.inv);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i] = Work<S>::load(rd[i * PL + q - cy(i) * RW - cx(i)], i, a.inv);
        }
        if (s == 1 && EDGE && t >= TAG_ZOUHE_FIRST) {
            // a boundary rule: listed; its gathered populations wait in the node's own slots
            list[atomicAdd(nlist, 1)] = (unsigned short)q;
#pragma unroll
            for (int i = 0; i < 9; ++i) wr[i * PL + q] = Work<S>::store(f[i], i, a.sc);
            continue;
        }
        tile_bulk<S, M>(a, t, X, Y, f);
        tile_store<S, SH, s, EDGE, M>(a, f, rd, wr, gd, go, X, Y, q, c >= E && c < WS - E && r >= E && r < HS - E);
    }
    if (EDGE) {
        if (s == 1) __syncthreads();
        const int n = s == 1 ? *nlist : listed;
        // the listed nodes, packed into warps from the block's last one down
#pragma unroll 1
        for (int e = SH::NT - 1 - (int)threadIdx.x; e < n; e += SH::NT) {
            const int q = list[e];
            const int c = q % RW, r = q / RW;
            if (c < O || c >= RW - O || r < O || r >= SH::RH - O) continue;
            const int X = x0 - (SH::T - 1) + c, Y = y0 - (SH::T - 1) + r;
            const int t = stag[q];
            Wk f[9];
#pragma unroll
            for (int i = 0; i < 9; ++i)
                f[i] = Work<S>::load(s == 1 ? wr[i * PL + q] : rd[i * PL + q - cy(i) * RW - cx(i)], i, a.inv);
            tile_boundary<S, SH, s, M, EXTRAP>(a, rd, t, X, Y, q, f);
            tile_store<S, SH, s, EDGE, M>(a, f, rd, wr, gd, (unsigned)(r - O) * pitch + (unsigned)(c - O) * (unsigned)sizeof(S), X, Y, q,
                                           c >= SH::T - 1 && c < RW - (SH::T - 1) && r >= SH::T - 1 && r < SH::RH - (SH::T - 1));
        }
    }
}

// Two nodes side by side, as one load or store of twice the width.  FP32 and 16-bit storage run pairs (FP32 172 -> 114 instructions
// an update, 134 -> 150 GLUPS at 8192 x 2048: addresses, loop and stores are shared and the arithmetic packed); FP64
// does not (its arithmetic is not packed, and two nodes' registers halve the resident warps: 66 -> 56 GLUPS).
template <class S>
__device__ __forceinline__ float2 pair_load(const S *p)            // p on a pair's boundary
{
    if constexpr (sizeof(S) == 4) return *reinterpret_cast<const float2 *>(p);
    else {
        const unsigned w = *reinterpret_cast<const unsigned *>(p);
        return make_float2(Half2Ops<S>::lo(w), Half2Ops<S>::hi(w));
    }
}

template <class S>
__device__ __forceinline__ float2 pair_gather(const S *p)          // p anywhere
{
    return make_float2(Work<S>::load(p[0], 0, 0.0f), Work<S>::load(p[1], 0, 0.0f));
}

// Direction i of the pair as stored; rs: its stochastic rounding bits (16-bit, RS).
template <class S, bool RS>
__device__ __forceinline__ void pair_store(S *p, float2 f, unsigned rs)
{
    if constexpr (sizeof(S) == 4) *reinterpret_cast<float2 *>(p) = f;
    else *reinterpret_cast<unsigned *>(p) = RS ? RsOps<S>::pack(f.x, f.y, rs) : Half2Ops<S>::pack(f.x, f.y);
}

// The rounding bits of nodes X, X + 1 of a row (rs_node, put): the bits of a quad's pair p are m (2 (9 p + i) + 1)
// with m the quad's hash times codec.cuh's constant; a pair that starts at an even X takes the upper
// half of one of them and the lower half of the next.
template <bool SPLIT>
struct PairBits {
    unsigned ma, oa, mb, ob;
    __device__ __forceinline__ unsigned bits(int i) const
    {
        const unsigned a = ma * (unsigned)(2 * i + 1) + oa;
        return SPLIT ? __byte_perm(a, mb * (unsigned)(2 * i + 1) + ob, 0x5432) : a;
    }
};

template <bool SPLIT>
__device__ __forceinline__ PairBits<SPLIT> pair_bits(const Geo &g, unsigned key, int X, int Y)
{
    const int q = (X - 1) & 3;          // 0 or 2; split pairs 1 or 3
    const unsigned row = (unsigned)Y * (unsigned)(g.lx + 2);
    PairBits<SPLIT> b;
    b.ma = rs_mix((row + (unsigned)(X - q)) ^ key) * 0x9e3779b9u;
    b.oa = (q & 2) ? 18u * b.ma : 0u;
    b.mb = SPLIT && q == 3 ? rs_mix((row + (unsigned)(X + 1)) ^ key) * 0x9e3779b9u : b.ma;
    b.ob = SPLIT && q == 1 ? 18u * b.ma : 0u;
    return b;
}

__device__ __forceinline__ unsigned long long x2(float2 v) { return *reinterpret_cast<unsigned long long *>(&v); }
__device__ __forceinline__ float2 f2(unsigned long long v) { return *reinterpret_cast<float2 *>(&v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x2(a)), "l"(x2(b)));
    return f2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x2(a)), "l"(x2(b)));
    return f2(d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x2(a)), "l"(x2(b)), "l"(x2(c)));
    return f2(d);
}
__device__ __forceinline__ float2 c2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, c2(-1.0f), a); }

// rules::bgk<float> on two nodes with the packed FP32 instructions: the same operations on the same
// operands in the same order, products fused where the compiler fuses them there (negated
// operands move a sign, which rounding to nearest does not see), so the same bits.
__device__ __forceinline__ void bgk_pair(float2 f[9], float omega)
{
    const float2 rho = add2(add2(add2(add2(f[0], f[1]), add2(f[2], f[3])), add2(add2(f[4], f[5]), add2(f[6], f[7]))), f[8]);
    const float2 inv = make_float2(__frcp_rn(rho.x), __frcp_rn(rho.y));
    const float2 jx = add2(add2(sub2(f[1], f[3]), sub2(f[5], f[6])), sub2(f[8], f[7]));
    const float2 jy = add2(add2(sub2(f[2], f[4]), sub2(f[5], f[8])), sub2(f[6], f[7]));
    const float2 ux = mul2(jx, inv), uy = mul2(jy, inv);
    const float2 base = fma2(c2(-1.5f), fma2(ux, ux, mul2(uy, uy)), c2(1.0f));
    const float2 n0 = mul2(c2(-4.f / 9.f), rho), n1 = mul2(c2(-1.f / 9.f), rho), n2 = mul2(c2(-1.f / 36.f), rho);
    const float2 nom = c2(-omega);
    f[0] = fma2(nom, fma2(n0, base, f[0]), f[0]);
#define LBGPU_RELAX2(I, J, N, CU)                                                     \
    {                                                                                 \
        const float2 cu = (CU);                                                       \
        const float2 ei = fma2(cu, fma2(c2(4.5f), cu, c2(3.0f)), base);               \
        const float2 ej = fma2(cu, fma2(c2(4.5f), cu, c2(-3.0f)), base);              \
        f[I] = fma2(nom, fma2(N, ei, f[I]), f[I]);                                    \
        f[J] = fma2(nom, fma2(N, ej, f[J]), f[J]);                                    \
    }
    LBGPU_RELAX2(1, 3, n1, ux)
    LBGPU_RELAX2(2, 4, n1, uy)
    LBGPU_RELAX2(5, 7, n2, add2(ux, uy))
    LBGPU_RELAX2(6, 8, n2, sub2(uy, ux))
#undef LBGPU_RELAX2
}

// bgk_offsets<false> on two nodes, in the same way.
__device__ __forceinline__ void bgk_offsets_pair(float2 D[9], float omega, float sc, float inv)
{
    const float2 sum = add2(add2(add2(add2(D[0], D[1]), add2(D[2], D[3])), add2(add2(D[4], D[5]), add2(D[6], D[7]))), D[8]);
    const float2 d = mul2(c2(inv), sum);
    const float2 Jx = add2(add2(sub2(D[1], D[3]), sub2(D[5], D[6])), sub2(D[8], D[7]));
    const float2 Jy = add2(add2(sub2(D[2], D[4]), sub2(D[5], D[8])), sub2(D[6], D[7]));
    const float2 ir = make_float2(__fdividef(1.0f, 1.0f + d.x), __fdividef(1.0f, 1.0f + d.y));
    const float2 q = mul2(c2(inv), ir);
    const float2 ux = mul2(Jx, q), uy = mul2(Jy, q);
    const float2 A = fma2(c2(-1.5f * inv), fma2(Jx, ux, mul2(Jy, uy)), d);
    const float2 ux45 = mul2(c2(4.5f * inv), ux), uy45 = mul2(c2(4.5f * inv), uy);
    const float om1 = 1.0f - omega;
    const float k0 = omega * sc * (4.f / 9.f), k1 = omega * sc * (1.f / 9.f), k2 = omega * sc * (1.f / 36.f);
    const float b1 = (3.0f * inv) * k1, b2 = (3.0f * inv) * k2;
    D[0] = fma2(c2(om1), D[0], mul2(c2(k0), A));
#define LBGPU_PAIR2(I, J, K, B, CU45, CJ)                             \
    {                                                                 \
        const float2 cj = (CJ);                                       \
        const float2 a = mul2(c2(K), fma2(CU45, cj, A));              \
        D[I] = fma2(c2(om1), D[I], fma2(c2(B), cj, a));               \
        D[J] = fma2(c2(om1), D[J], fma2(c2(-(B)), cj, a));            \
    }
    LBGPU_PAIR2(1, 3, k1, b1, ux45, Jx)
    LBGPU_PAIR2(2, 4, k1, b1, uy45, Jy)
    LBGPU_PAIR2(5, 7, k2, b2, add2(ux45, uy45), add2(Jx, Jy))
    LBGPU_PAIR2(6, 8, k2, b2, sub2(uy45, ux45), sub2(Jy, Jx))
#undef LBGPU_PAIR2
}

// bgk_offsets<true> on two nodes of a row.
__device__ __forceinline__ void bgk_offsets_pair_shifted(float2 D[9], float omega, float sc, float inv, float us)
{
    const float2 sum = add2(add2(add2(add2(D[0], D[1]), add2(D[2], D[3])), add2(add2(D[4], D[5]), add2(D[6], D[7]))), D[8]);
    const float2 d = mul2(c2(inv), sum);
    const float2 Jx = add2(add2(sub2(D[1], D[3]), sub2(D[5], D[6])), sub2(D[8], D[7]));
    const float2 Jy = add2(add2(sub2(D[2], D[4]), sub2(D[5], D[8])), sub2(D[6], D[7]));
    const float2 ir = make_float2(__fdividef(1.0f, 1.0f + d.x), __fdividef(1.0f, 1.0f + d.y));
    const float2 q = mul2(c2(inv), ir);
    const float2 ux = fma2(Jx, q, mul2(c2(us), ir)), uy = mul2(Jy, q);
    const float2 t = sub2(ux, c2(us));
    const float2 A = fma2(c2(-1.5f * us), t, fma2(c2(-1.5f * inv), fma2(Jx, ux, mul2(Jy, uy)), d));
    const float2 ux45 = mul2(c2(4.5f * inv), ux), uy45 = mul2(c2(4.5f * inv), uy);
    const float hs = 4.5f * us;
    const float2 A1 = fma2(c2(hs), t, A), ev = mul2(c2(hs), uy);
    const float2 A5 = add2(A1, ev), A6 = sub2(A1, ev);
    const float om1 = 1.0f - omega;
    const float k0 = omega * sc * (4.f / 9.f), k1 = omega * sc * (1.f / 9.f), k2 = omega * sc * (1.f / 36.f);
    const float b1 = (3.0f * inv) * k1, b2 = (3.0f * inv) * k2;
    D[0] = fma2(c2(om1), D[0], mul2(c2(k0), A));
#define LBGPU_PAIR2S(I, J, K, B, CU45, CJ, AP)                        \
    {                                                                 \
        const float2 cj = (CJ);                                       \
        const float2 a = mul2(c2(K), fma2(CU45, cj, AP)), b = mul2(c2(B), cj); \
        D[I] = fma2(c2(om1), D[I], add2(a, b));                       \
        D[J] = fma2(c2(om1), D[J], sub2(a, b));                       \
    }
    LBGPU_PAIR2S(1, 3, k1, b1, ux45, Jx, A1)
    LBGPU_PAIR2S(2, 4, k1, b1, uy45, Jy, A)
    LBGPU_PAIR2S(5, 7, k2, b2, add2(ux45, uy45), add2(Jx, Jy), A5)
    LBGPU_PAIR2S(6, 8, k2, b2, sub2(uy45, ux45), sub2(Jy, Jx), A6)
#undef LBGPU_PAIR2S
}

// Step s of a tile that holds no perimeter node and no boundary rule, two nodes a thread (FP32 and 16-bit).
// The pairs of step s start at column x0 - (T - s): a step later they start one column on, so the
// two populations that a pair takes from x - 1 or x + 1 were stored (or, T being even, lie in the
// planes) as one pair, and only those of the three directions along y are read one by one.
// Step 1 sets *met where it meets a node with a boundary rule, which it does not apply.
template <class S, class SH, int s, int M>
__device__ __forceinline__ void tile_step_pairs(const TileArgs<S> &a, S *__restrict__ sm, uint8_t *__restrict__ stag,
                                                int *__restrict__ met, int x0, int y0)
{
    constexpr bool RS = (M & TILE_RS) != 0, SHIFT = (M & TILE_SHIFT) != 0;
    constexpr int E = SH::T - s, WP = (SH::W + 2 * E) / 2, HS = SH::H + 2 * E, O = s - 1, RW = SH::RW, PL = SH::PL;
    const Geo &g = a.g;
    const S *rd = sm + (size_t)(s & 1) * (SH::NBUF - 1) * SH::B1;
    S *wr = sm + (size_t)((s - 1) & 1) * (SH::NBUF - 1) * SH::B1;
    const long long o0 = (long long)(y0 - E) * g.pitch + (x0 - E + g.xoff - 1);
    const unsigned pitch = (unsigned)g.pitch * (unsigned)sizeof(S);
    int c = (int)threadIdx.x % WP, r = (int)threadIdx.x / WP;
#pragma unroll 1
    for (; r < HS; c += SH::NT % WP, r += SH::NT / WP, r += c >= WP ? 1 : 0, c -= c >= WP ? WP : 0) {
        const int q = (r + O) * RW + (2 * c + O);
        const unsigned go = (unsigned)r * pitch + (unsigned)c * (unsigned)(2 * sizeof(S));
        float2 f[9];
        unsigned t;
        if (s == 1) {
            const uint8_t *gt = a.tag + o0 + (go / (unsigned)sizeof(S));
            t = gt[0] | ((unsigned)gt[1] << 8);
            const char *gs = reinterpret_cast<const char *>(a.src + o0) + go;
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const S *p = reinterpret_cast<const S *>(gs + ((long long)i * g.plane - (long long)cy(i) * g.pitch) * (long long)sizeof(S)) - cx(i);
                f[i] = cx(i) != 0 ? pair_load(p) : pair_gather(p);
            }
            *reinterpret_cast<unsigned short *>(stag + q) = (unsigned short)t;
        } else {
            t = stag[q] | ((unsigned)stag[q + 1] << 8);
            const S *p = rd + q;
#pragma unroll
            for (int i = 0; i < 9; ++i)
                f[i] = cx(i) != 0 ? pair_load(p + (i * PL - cy(i) * RW - cx(i))) : pair_gather(p + (i * PL - cy(i) * RW));
        }
        if (t == 0x0101u) {
            if constexpr (SHIFT) bgk_offsets_pair_shifted(f, a.omega_f, a.sc, a.inv, g.shift_u[y0 - E + r]);
            else if constexpr (sizeof(S) == 2) bgk_offsets_pair(f, a.omega_f, a.sc, a.inv);
            else bgk_pair(f, a.omega_f);
        } else {
            if (s == 1 && ((t & 0xffu) >= TAG_ZOUHE_FIRST || (t >> 8) >= TAG_ZOUHE_FIRST)) *met = 1;
            float h[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) h[i] = f[i].x;
            tile_bulk<S, M>(a, (int)(t & 0xffu), x0 - E + 2 * c, y0 - E + r, h);
#pragma unroll
            for (int i = 0; i < 9; ++i) { f[i].x = h[i]; h[i] = f[i].y; }
            tile_bulk<S, M>(a, (int)(t >> 8), x0 - E + 2 * c + 1, y0 - E + r, h);
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i].y = h[i];
        }
        if (SHIFT && g.shift_rebased(y0 - E + r)) {
            const float *rebase = g.shift_rebase(y0 - E + r);
#pragma unroll
            for (int i = 0; i < 9; ++i)
                if (cy(i) != 0) f[i] = add2(f[i], mul2(c2(rebase[i]), c2(a.sc)));
        }
        constexpr bool SPLIT = (E & 1) != 0;              // x0 is odd: X = x0 - E + 2 c is even
        PairBits<SPLIT> b = {};
        if constexpr (RS) b = pair_bits<SPLIT>(g, a.keys[s - 1], x0 - E + 2 * c, y0 - E + r);
        if (s == SH::T) {
            char *gd = reinterpret_cast<char *>(a.dst + o0) + go;
#pragma unroll
            for (int i = 0; i < 9; ++i)
                pair_store<S, RS>(reinterpret_cast<S *>(gd + (long long)i * g.plane * (long long)sizeof(S)), f[i], RS ? b.bits(i) : 0u);
        } else {
#pragma unroll
            for (int i = 0; i < 9; ++i) pair_store<S, RS>(wr + i * PL + q, f[i], RS ? b.bits(i) : 0u);
        }
    }
}

// Steps s to T; false where step 1 of a tile off the perimeter met a boundary rule: nothing is written to the planes
// yet, and the tile takes its steps afresh as one with rules.
template <class S, class SH, int s, bool EDGE, int M, bool EXTRAP>
__device__ __forceinline__ bool tile_steps(const TileArgs<S> &a, S *sm, uint8_t *stag, unsigned short *list, int *nlist,
                                           int x0, int y0)
{
    if constexpr (!EDGE && sizeof(S) <= 4) tile_step_pairs<S, SH, s, M>(a, sm, stag, nlist, x0, y0);
    else tile_step<S, SH, s, EDGE, M, EXTRAP>(a, sm, stag, list, nlist, x0, y0);
    if constexpr (s < SH::T) {
        __syncthreads();
        if (s == 1 && !EDGE && sizeof(S) <= 4 && a.rules_inside && *nlist != 0) return false;
        return tile_steps<S, SH, s + 1, EDGE, M, EXTRAP>(a, sm, stag, list, nlist, x0, y0);
    }
    return true;
}

// The T steps of the tile at (x0, y0) by one block.
template <class SH, int M, bool EXTRAP>
__device__ __forceinline__ void tile_block(const TileArgs<typename SH::S> &a, unsigned char *smem, int x0, int y0)
{
    using S = typename SH::S;
    S *sm = reinterpret_cast<S *>(smem);
    uint8_t *stag = smem + SH::POPS;
    unsigned short *list = reinterpret_cast<unsigned short *>(stag + SH::TAGS);
    int *nlist = reinterpret_cast<int *>(smem + SH::SMEM - 16);
    constexpr int E = SH::T - 1;
    // Where some node off the perimeter has a boundary rule, pairs (FP32 and 16-bit) find out in step 1 whether it is one
    // of this tile's; FP64, whose two forms run alike, does not try.
    const bool inside = (sizeof(S) <= 4 || !a.rules_inside) &&
                        x0 - E >= 2 && x0 + SH::W - 1 + E <= a.g.lx - 1 && y0 - E >= 2 && y0 + SH::H - 1 + E <= a.g.ly - 1;
    if (inside) {
        if (a.rules_inside) {
            if (threadIdx.x == 0) *nlist = 0;
            __syncthreads();
        }
        if (tile_steps<S, SH, 1, false, M, EXTRAP>(a, sm, stag, list, nlist, x0, y0)) return;
        __syncthreads();           // every thread has read what it met
    }
    if (threadIdx.x == 0) *nlist = 0;
    __syncthreads();
    tile_steps<S, SH, 1, true, M, EXTRAP>(a, sm, stag, list, nlist, x0, y0);
}

template <class SH, int M, bool EXTRAP>
__global__ void __launch_bounds__(SH::NT, SH::MINB) k_tile(const __grid_constant__ TileArgs<typename SH::S> a)
{
    extern __shared__ __align__(16) unsigned char tile_smem[];
    if constexpr (SH::W % 16 == 0) {         // (a prefetch is of whole 16-byte units)
        if (a.pf > 0 && threadIdx.x < 9 * SH::H && blockIdx.x + (unsigned)a.pf < gridDim.x) {
            int px, py;
            tile_place(blockIdx.x + (unsigned)a.pf, a.nx, a.ny, a.ring_first, px, py);
            const int Yp = 1 + py * SH::H + (int)threadIdx.x % SH::H, Xp = a.x_first + px * SH::W;
            if (Yp <= a.g.ly && Xp >= 1 && Xp + SH::W - 1 <= a.g.lx)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(plane(a.src, a.g, (int)threadIdx.x / SH::H) + a.g.idx(Xp, Yp)),
                             "n"(SH::W * (int)sizeof(typename SH::S)) : "memory");
        }
    }
    int tx, ty;
    tile_place(blockIdx.x, a.nx, a.ny, a.ring_first, tx, ty);
    tile_block<SH, M, EXTRAP>(a, tile_smem, a.x_first + tx * SH::W, 1 + ty * SH::H);
}

// T steps of every tile of a batch's work list (x0, y0: the tile's first node): launch `unit` of a
// chunk, so a member's state is where `unit` launches have taken it from its descriptor's.
template <class SH, bool RS>
__global__ void __launch_bounds__(SH::NT, SH::MINB) k_batch_tile(const BatchInst *__restrict__ insts,
                                                                 const BatchWork *__restrict__ work, int unit)
{
    using S = typename SH::S;
    extern __shared__ __align__(16) unsigned char tile_smem[];
    const BatchWork it = work[blockIdx.x];
    const BatchInst &d = insts[it.inst];
    TileArgs<S> a;
    a.g = d.g;
    const int src = d.cur0 ^ (unit & 1), pa = d.tau0 & 1;      // T is even: step 1's parity is the descriptor's
    a.src = static_cast<const S *>(d.buf[src]);
    a.dst = static_cast<S *>(d.buf[src ^ 1]);
    a.tag = d.tag;
    a.bc = d.bc;
    a.zgb = nullptr;
    a.omega = d.omega;
    a.omega_f = (float)d.omega;
    const size_t slot = 9 * (size_t)d.g.nper;
    const int now = batch_side_slot(d.side_slot, pa), last = batch_side_slot(d.side_slot, pa ^ 1);
    const int spare = sizeof(S) == 2 ? now ^ 2 : 3 - now - last;              // side_other
    S *side = static_cast<S *>(d.side);
    a.stale1 = side + slot * ((unit & 1) ? spare : now);
    a.out_prev = side + slot * ((unit & 1) ? now : spare);
    a.out_last = side + slot * last;
    a.sc = d.scale;
    a.inv = d.inv_scale;
    a.x_first = 1;
    a.rules_inside = d.rules_inside;
    if constexpr (RS) {
        if (d.rs) {
#pragma unroll
            for (int k = 0; k < SH::T; ++k) a.keys[k] = rs_key(d.rs_seed, (unsigned long long)(d.tau0 + unit * SH::T + k));
            tile_block<SH, 1, false>(a, tile_smem, it.x0, it.y0);
            return;
        }
    }
    tile_block<SH, 0, false>(a, tile_smem, it.x0, it.y0);
}
