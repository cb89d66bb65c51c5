// node.cuh -- per-node device functions shared by the kernels (kernels.cu, tile.cu): addressing, the
// post-stream value of a slot, stored and working values, the collision of a node.
#pragma once
#include "codec.cuh"
#include "kernels.h"
#include "lbgpu.h"

namespace lbgpu {

namespace {

constexpr int BX = 128;  // threads along x per block (coalesced axis)

template <class S>
__device__ __forceinline__ const S *plane(const S *b, const Geo &g, int i)
{
    return b + (size_t)i * (size_t)g.plane;
}
template <class S>
__device__ __forceinline__ S *plane(S *b, const Geo &g, int i)
{
    return b + (size_t)i * (size_t)g.plane;
}

// Table entry (p0, p1) of a boundary node: (ux, uy) or (rho, uPar).
__device__ __forceinline__ void node_params(const double *__restrict__ bc, int nb, int t, int X, int Y,
                                            double &p0, double &p1)
{
    p0 = 0.0; p1 = 0.0;
    if (t >= TAG_ZOUHE_FIRST && t < TAG_COUNT) {
        const int tb = tag_table(t);
        const int coord = (tag_side(t) <= SIDE_LOWER) ? X : Y;
        p0 = bc[(tb * 2 + 0) * nb + coord];
        p1 = bc[(tb * 2 + 1) * nb + coord];
    }
}

__device__ __forceinline__ void node_params(const double *__restrict__ bc, const Geo &g, int t,
                                            int X, int Y, double &p0, double &p1)
{
    node_params(bc, g.nb, t, X, Y, p0, p1);
}

template <class S, bool EXACT = false>
__device__ __forceinline__ void collide_node(const double *__restrict__ bc, const Geo &g, int t,
                                             int X, int Y, typename Codec<S>::R f[9], double omega)
{
    using R = typename Codec<S>::R;
    double p0, p1;
    node_params(bc, g, t, X, Y, p0, p1);
    rules::collide<R, EXACT>(t, f, (R)omega, (R)p0, (R)p1);
}

template <class S>
__device__ __forceinline__ typename Codec<S>::R dec_row(const Geo &g, S v, int i, float inv, int Y);

// Where the post-stream value of slot i at node (X, Y) lies, any node of the lattice including the ghost
// ring, under each view (kernels.h).  Ghost slots that no interior node streams into keep the
// content of the buffer the state lives in, as in the reference: for the pull scheme `other`
// is the second buffer; for the AA scheme's swapped view (an odd step count, which the
// reference leaves in its second buffer) `other` is that buffer's saved ghost ring
// [9][nghost].
template <class S>
__device__ __forceinline__ const S *logical_at(const Geo &g, int view, const S *__restrict__ cur, const S *__restrict__ other,
                                               const S *__restrict__ side, int X, int Y, int i)
{
    const int sx = X - cx(i), sy = Y - cy(i);
    const bool streamed = g.interior(sx, sy), inside = g.interior(X, Y);
    const S *stale = side + ((size_t)i * g.nper + g.pidx(X, Y));
    switch (view) {
    case VIEW_PULL_PENDING: return streamed ? plane(cur, g, i) + g.idx(sx, sy) : (inside ? stale : plane(other, g, i) + g.idx(X, Y));
    case VIEW_AA_NATURAL: return inside && !streamed ? stale : plane(cur, g, i) + g.idx(X, Y);
    case VIEW_AA_SWAPPED:
        return streamed ? plane(cur, g, opp(i)) + g.idx(sx, sy) : (inside ? stale : other + ((size_t)i * g.nghost() + g.gidx(X, Y)));
    default: return plane(cur, g, i) + g.idx(X, Y);
    }
}

// The nine slots of a node: their addresses first, so that all nine loads are in flight.
template <class S>
__device__ __forceinline__ void logical_node(const Geo &g, int view, const S *__restrict__ cur, const S *__restrict__ other,
                                             const S *__restrict__ side, int X, int Y, float inv, typename Codec<S>::R f[9])
{
    const S *at[9];
    S v[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) at[i] = logical_at(g, view, cur, other, side, X, Y, i);
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = *at[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) f[i] = dec_row<S>(g, v[i], i, inv, Y);
}

// ---- 16-bit storage, four nodes per thread ------------------------------------------------
//
// Stored value D_i = (f_i - w_i) 2^s.  With sum(w) = 1 and sum(c w) = 0 the BGK step works on
// D directly: rho = 1 + 2^-s sum(D), j = 2^-s sum(c D), and
//   D_i' = D_i + omega (E_i - D_i),  E_i = 2^s w_i (rho (1 + 3 cu + 4.5 cu^2 - 1.5 u^2) - 1),
// so there is no per-population decode or encode arithmetic, only the conversions (two per
// instruction when packing).  Boundary rules decode to f and use the generic path.

template <class S> struct Half2Ops;
template <> struct Half2Ops<__half> {
    static __device__ __forceinline__ float lo(unsigned w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
    static __device__ __forceinline__ float hi(unsigned w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }
    static __device__ __forceinline__ unsigned pack(float a, float b)
    {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const unsigned *>(&h);
    }
};
template <> struct Half2Ops<__nv_bfloat16> {
    static __device__ __forceinline__ float lo(unsigned w) { return __uint_as_float(w << 16); }
    static __device__ __forceinline__ float hi(unsigned w) { return __uint_as_float(w & 0xffff0000u); }
    static __device__ __forceinline__ unsigned pack(float a, float b)
    {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const unsigned *>(&h);
    }
};

// BGK on scaled offsets D[9] of one node (sc = 2^s, inv = 2^-s).  With d = rho - 1 =
// inv sum(D) and j = rho u = inv sum(c D), rho c.u = c.j and rho u^2 = j.u give
//   E_i = sc w_i (A + 3 c.j + 4.5 (c.u)(c.j)),  A = d - 1.5 j.u,
// and the relaxation is D_i' = (1 - omega) D_i + omega E_i.  Opposite directions i, opp(i)
// share c.u and c.j up to sign: omega E_i, omega E_opp = a +- b with
// a = k (A + 4.5 (c.u)(c.j)), b = 3 k c.j, k = omega sc w.
// With a row shift (SHIFT, offsets relative to S_i = f_eq_i(1, (us, 0)) instead of w_i):
// j = (us, 0) + inv J, E_i = sc (f_eq_i(rho, u) - S_i), so A gains -1.5 us (ux - us) and a gains
// 4.5 k (c.us)(c.u - c.us); b is unchanged.  Without it the arithmetic is exactly the unshifted one.
// 1/rho uses the hardware reciprocal (the 16-bit path is held to a tolerance, not bit-exact).
template <bool SHIFT>
__device__ __forceinline__ void bgk_offsets(float D[9], float omega, float sc, float inv, float us)
{
    // J = 2^s (j - us): scaled sums; u = J inv / rho (+ us / rho), inv folded into constants
    const float sum = ((D[0] + D[1]) + (D[2] + D[3])) + ((D[4] + D[5]) + (D[6] + D[7])) + D[8];
    const float d = inv * sum;
    const float Jx = (D[1] - D[3]) + (D[5] - D[6]) + (D[8] - D[7]);
    const float Jy = (D[2] - D[4]) + (D[5] - D[8]) + (D[6] - D[7]);
    const float ir = __fdividef(1.0f, 1.0f + d);
    const float q = inv * ir;
    const float ux = SHIFT ? fmaf(Jx, q, __fmul_rn(us, ir)) : Jx * q, uy = Jy * q;
    float A = fmaf(-1.5f * inv, fmaf(Jx, ux, Jy * uy), d);
    // shifted terms: t = ux - us; 4.5 (c.us)(c.u - c.us) is e1 = 4.5 us t for (1, 3) and
    // e1 +- 4.5 us uy for (5, 7) and (6, 8), folded into the pair's constant term: A1 = A + e1,
    // A1 +- 4.5 us uy
    const float t = SHIFT ? __fsub_rn(ux, us) : 0.0f;
    if (SHIFT) A = fmaf(-1.5f * us, t, A);
    const float ux45 = (4.5f * inv) * ux, uy45 = (4.5f * inv) * uy;
    const float hs = 4.5f * us;
    const float A1 = SHIFT ? fmaf(hs, t, A) : A, ev = SHIFT ? __fmul_rn(hs, uy) : 0.0f;
    const float A5 = SHIFT ? __fadd_rn(A1, ev) : A, A6 = SHIFT ? __fsub_rn(A1, ev) : A;
    const float om1 = 1.0f - omega;
    const float k0 = omega * sc * (4.f / 9.f), k1 = omega * sc * (1.f / 9.f), k2 = omega * sc * (1.f / 36.f);
    D[0] = fmaf(om1, D[0], k0 * A);
    // The shifted terms use explicitly rounded operations: no multiply-add contraction may
    // differ between the kernels that inline this, so every scheme stays bit-identical.
#define LBGPU_PAIR(I, J, K, CU45, CJ, AP)                              \
    {                                                                  \
        const float cj = (CJ);                                         \
        if (SHIFT) {                                                   \
            const float a = __fmul_rn(K, fmaf(CU45, cj, (AP)));        \
            const float b = __fmul_rn((3.0f * inv) * K, cj);          \
            D[I] = fmaf(om1, D[I], __fadd_rn(a, b));                   \
            D[J] = fmaf(om1, D[J], __fsub_rn(a, b));                   \
        } else {                                                       \
            const float a = K * fmaf(CU45, cj, A);                     \
            const float b = ((3.0f * inv) * K) * cj;                   \
            D[I] = fmaf(om1, D[I], a + b);                             \
            D[J] = fmaf(om1, D[J], a - b);                             \
        }                                                              \
    }
    LBGPU_PAIR(1, 3, k1, ux45, Jx, A1)
    LBGPU_PAIR(2, 4, k1, uy45, Jy, A)
    LBGPU_PAIR(5, 7, k2, __fadd_rn(ux45, uy45), __fadd_rn(Jx, Jy), A5)
    LBGPU_PAIR(6, 8, k2, __fsub_rn(uy45, ux45), __fsub_rn(Jy, Jx), A6)
#undef LBGPU_PAIR
}


// Working values of a kernel: decoded populations f for FP64/FP32, the stored offsets D as
// float for 16-bit storage (see bgk_offsets); collide_w applies a node's rule to them.  Every
// kernel of one storage type uses these, so all schemes agree bit for bit.
template <class S> struct Work {
    using W = typename Codec<S>::R;
    static __device__ __forceinline__ W load(S v, int i, float inv) { return Codec<S>::dec(v, i, inv); }
    static __device__ __forceinline__ S store(W w, int i, float sc) { return Codec<S>::enc(w, i, sc); }
};
template <> struct Work<__half> {
    using W = float;
    static __device__ __forceinline__ float load(__half v, int, float) { return __half2float(v); }
    static __device__ __forceinline__ __half store(float w, int, float) { return __float2half_rn(w); }
};
template <> struct Work<__nv_bfloat16> {
    using W = float;
    static __device__ __forceinline__ float load(__nv_bfloat16 v, int, float) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 store(float w, int, float) { return __float2bfloat16_rn(w); }
};

// Stochastic rounding (codec.cuh) is a compile-time choice of a kernel (RS), so no store
// carries a branch: RS kernels run only for 16-bit lattices with it on, whose collision key is
// then never 0.
// The random word of node (X, Y) for a collision key.
template <class S, bool RS>
__device__ __forceinline__ RsNode rs_node(const Geo &g, unsigned key, int X, int Y)
{
    if constexpr (RS && sizeof(S) == 2) {
        const int q = (X - 1) & 3;
        return RsNode{rs_mix(((unsigned)Y * (unsigned)(g.lx + 2) + (unsigned)(X - q)) ^ key), q};
    }
    return RsNode{0u, 0};
}

// A post-collision working value of direction i as stored: rounded to nearest, or (RS)
// stochastically with the node's random word h.
template <class S, bool RS>
__device__ __forceinline__ S put(typename Work<S>::W w, int i, float sc, RsNode h)
{
    if constexpr (RS && sizeof(S) == 2) {
        const unsigned p = rs_pair(h.hq, h.q >> 1, i);
        return RsOps<S>::one(w, (h.q & 1) ? (p >> 16) : p);
    }
    return Work<S>::store(w, i, sc);
}

// Decode / encode of a value consumed at row Y (read-outs, uploads, initial states).
template <class S>
__device__ __forceinline__ typename Codec<S>::R dec_row(const Geo &g, S v, int i, float inv, int Y)
{
    if constexpr (sizeof(S) == 2) {
        if (g.shift_u) return fmaf(Work<S>::load(v, i, inv), inv, g.shift_base(Y)[i]);
    }
    return Codec<S>::dec(v, i, inv);
}

template <class S>
__device__ __forceinline__ S enc_row(const Geo &g, typename Codec<S>::R f, int i, float sc, int Y)
{
    if constexpr (sizeof(S) == 2) {
        if (g.shift_u) return Work<S>::store(__fmul_rn(__fsub_rn(f, g.shift_base(Y)[i]), sc), i, sc);
    }
    return Codec<S>::enc(f, i, sc);
}

// The post-stream state of interior node (X, Y) under a view, decoded: logical_node(), but off the perimeter, where
// every slot has an interior source, without its tests.
template <class S>
__device__ __forceinline__ void load_state(const Geo &g, int view, const S *__restrict__ cur, const S *__restrict__ other,
                                           const S *__restrict__ side, int X, int Y, float inv,
                                           typename Codec<S>::R f[9])
{
    if (g.perimeter(X, Y)) {
        logical_node(g, view, cur, other, side, X, Y, inv, f);
        return;
    }
    const long long o = g.idx(X, Y);
    S v[9];
    if (view == VIEW_PULL_PENDING) {
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = plane(cur, g, i)[o - cx(i) - (long long)cy(i) * g.pitch];
    } else if (view == VIEW_AA_SWAPPED) {
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = plane(cur, g, opp(i))[o - cx(i) - (long long)cy(i) * g.pitch];
    } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = plane(cur, g, i)[o];
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) f[i] = dec_row<S>(g, v[i], i, inv, Y);
}

// A post-collision value of direction i at row Y, as stored in a population plane: with a row
// shift it is relative to the row that consumes it after streaming, Y + c_iy (stale-slot copies
// in the side store are consumed by the node itself and stay relative to row Y).
// SH: 0 no shift, 1 shift (known at compile time), 2 decided by g.shift_u at run time.
// Rows whose rebase values are all zero (shift_rebased false) store unchanged in every kernel.
template <class S, int SH = 2>
__device__ __forceinline__ typename Work<S>::W stored_out(const Geo &g, int Y, int i, typename Work<S>::W w,
                                                          float sc)
{
    if constexpr (sizeof(S) == 2 && SH != 0) {
        if (cy(i) != 0 && (SH == 1 || g.shift_u) && g.shift_rebased(Y))
            return __fadd_rn(w, __fmul_rn(g.shift_rebase(Y)[i], sc));
    }
    return w;
}

// A non-BGK rule on one node's 16-bit offsets: decode, the generic rule, encode.  Out of line so
// the bulk path keeps its registers (it runs for boundary and obstacle nodes only); the shifted
// form is a separate function, because a larger callee costs the 64-register quad kernel spills.
template <class S>
static __device__ __noinline__ void boundary_offsets(const double *__restrict__ bc, Geo g, int t, int X,
                                                     int Y, float D[9], double omega, float sc, float inv)
{
    float f[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) f[i] = fmaf(D[i], inv, wgtf(i));
    collide_node<S>(bc, g, t, X, Y, f, omega);
#pragma unroll
    for (int i = 0; i < 9; ++i) D[i] = (f[i] - wgtf(i)) * sc;
}

// The same with offsets from the row's shift equilibrium (base: S_i of the row).
template <class S>
static __device__ __noinline__ void boundary_offsets_shifted(const double *__restrict__ bc, int nb,
                                                             const float *__restrict__ base, int t, int X, int Y,
                                                             float D[9], double omega, float sc, float inv)
{
    float f[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) f[i] = fmaf(D[i], inv, base[i]);
    double p0, p1;
    node_params(bc, nb, t, X, Y, p0, p1);
    rules::collide<float>(t, f, (float)omega, (float)p0, (float)p1);
#pragma unroll
    for (int i = 0; i < 9; ++i) D[i] = (f[i] - base[i]) * sc;
}

template <class S, int SH = 2>
__device__ __forceinline__ void collide_w(const double *__restrict__ bc, const Geo &g, int t, int X,
                                          int Y, typename Work<S>::W w[9], double omega, float sc,
                                          float inv)
{
    if constexpr (sizeof(S) == 2) {
        if (t == TAG_BGK) {
            if constexpr (SH == 1) bgk_offsets<true>(w, (float)omega, sc, inv, g.shift_u[Y]);
            else if constexpr (SH == 0) bgk_offsets<false>(w, (float)omega, sc, inv, 0.0f);
            else if (g.shift_u) bgk_offsets<true>(w, (float)omega, sc, inv, g.shift_u[Y]);
            else bgk_offsets<false>(w, (float)omega, sc, inv, 0.0f);
        } else {
            float tmp[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) tmp[i] = w[i];
            if (SH == 1 || (SH == 2 && g.shift_u))
                boundary_offsets_shifted<S>(bc, g.nb, g.shift_base(Y), t, X, Y, tmp, omega, sc, inv);
            else
                boundary_offsets<S>(bc, g, t, X, Y, tmp, omega, sc, inv);
#pragma unroll
            for (int i = 0; i < 9; ++i) w[i] = tmp[i];
        }
    } else {
        collide_node<S>(bc, g, t, X, Y, w, omega);
    }
}

// collide_w of a boundary node whose table entry is given (p0, p1) instead of read.
template <class S>
__device__ __forceinline__ void collide_given(const Geo &g, int t, typename Work<S>::W w[9], double omega, float sc,
                                              float inv, double p0, double p1)
{
    using R = typename Codec<S>::R;
    R f[9];
    if constexpr (sizeof(S) == 2) {
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = fmaf(w[i], inv, wgtf(i));
        rules::collide<R>(t, f, (R)omega, (R)p0, (R)p1);
#pragma unroll
        for (int i = 0; i < 9; ++i) w[i] = (f[i] - wgtf(i)) * sc;
    } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = w[i];
        rules::collide<R>(t, f, (R)omega, (R)p0, (R)p1);
#pragma unroll
        for (int i = 0; i < 9; ++i) w[i] = f[i];
    }
}

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

template <class S> S *B(const DevLattice &d, int b) { return static_cast<S *>(d.buf[b]); }
// The `other` argument of logical_at(): the pull scheme's second buffer, or the AA ring copy.
template <class S> S *OTHER(const DevLattice &d, int cur)
{
    return d.buf[1] ? static_cast<S *>(d.buf[(1 - cur) ^ d.ghost_flip]) : static_cast<S *>(d.ghost2);
}
// A slot of the side store; a parity's.
template <class S> S *SIDE_SLOT(const DevLattice &d, int slot)
{
    return static_cast<S *>(d.side) + (size_t)slot * 9 * (size_t)d.g.nper;
}
template <class S> S *SIDE(const DevLattice &d, int p) { return SIDE_SLOT<S>(d, d.side_slot[p & 1]); }

}  // namespace

// Run F<S>() with S the lattice's storage type.
#define LBGPU_DISPATCH(d, BODY)                                        \
    switch ((d).precision) {                                          \
    case LBGPU_F64: { using S = double; BODY; } break;                \
    case LBGPU_F32: { using S = float; BODY; } break;                 \
    case LBGPU_F16: { using S = __half; BODY; } break;                \
    default: { using S = __nv_bfloat16; BODY; } break;                \
    }

}  // namespace lbgpu
