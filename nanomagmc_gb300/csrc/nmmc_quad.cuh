// Four consecutive same-colour Heisenberg sites of one row as two packed FP32 pairs.
//
// The scalar form of the four-site half-sweep issued 169 thread-instructions per update (36 of
// them 32 x 32 -> 64-bit multiplies and exclusive-ors of the generator) and ran at 64 % of the
// issue rate with DRAM 55 % busy. Here the per-site FP32 work of two sites shares the packed
// instructions of this architecture (fma/add/mul.rn.f32x2: one issue slot for two IEEE
// operations): 138 per update. What is left is bound by the two dispatch ports of the FMA-heavy
// pipe (the multiplies take four cycles each, a packed operation two; 69 % busy) and of the
// ALU. Each half of a packed operation rounds exactly like the scalar one, and the operations
// and their order per site are those of heis_field and heis_try, so the chain is the same bit
// for bit. Benchmark half-sweep (40 chains of 128^3): 272 -> 243 us.
#pragma once
#include "nmmc_kernels.cuh"

namespace nmmc {

// Spins of a quad in one component: sites (0, 1) and (2, 3).
struct F2x2 { f2 a, b; };

// A quad at `off` floats past a plane's base (16-byte aligned). The base is the same for every
// thread of a block and the offset 32 bits, so that an access needs one address register and
// no 64-bit arithmetic of its own.
__device__ __forceinline__ F2x2 ld_quad(const float* base, uint32_t off) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(reinterpret_cast<const char*>(base) + off * 4u);
    return F2x2{{t.x}, {t.y}};
}
__device__ __forceinline__ void st_quad(float* base, uint32_t off, const F2x2& v) {
    *reinterpret_cast<ulonglong2*>(reinterpret_cast<char*>(base) + off * 4u) = make_ulonglong2(v.a.v, v.b.v);
}
__device__ __forceinline__ F2x2 zero_quad() { return F2x2{{0ull}, {0ull}}; }

// The x-neighbours of a quad that are not its same-index sites: compact indices h0+1 .. h0+4
// (xp = 1) or h0-1 .. h0+2 (xp = 0); `ex` is the one outside the quad (0 where absent).
__device__ __forceinline__ F2x2 shifted_quad(const F2x2& same, float ex, bool xp) {
    const float s0 = lo(same.a), s1 = hi(same.a), s2 = lo(same.b), s3 = hi(same.b);
    return F2x2{pk(xp ? s1 : ex, xp ? s2 : s0), pk(xp ? s3 : s1, xp ? ex : s2)};
}

// Adds one axis' terms of the local field to h (and, with EF, of its DMI part to d) for a pair
// of sites whose +axis and -axis neighbours are P and M: the operations of heis_field for that
// axis, in its order; d takes the DMI's of them alone. For the +-pair kinds the sign `flip` (axis 0
// only) swaps the two neighbours' roles: their sum is symmetric and their difference changes sign,
// so it is folded into the DMI strength and the neighbours need not be sorted by direction.
template <int DK, int A, bool EF>
__device__ __forceinline__ void axis_terms(const DevModel& m, const f2 (&P)[3], const f2 (&M)[3], float flip,
                                           f2 (&h)[3], f2 (&d)[3]) {
    constexpr int kp = 2 * A, km = 2 * A + 1;
    if (DK <= kDmiGeneral) {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int k = side ? km : kp;
            const f2(&n)[3] = side ? M : P;
            const f2 J = pk(m.J[k], m.J[k]);
            h[0] = fma2(J, n[0], h[0]);
            h[1] = fma2(J, n[1], h[1]);
            h[2] = fma2(J, n[2], h[2]);
            if (DK == kDmiGeneral) {
                const f2 D0 = pk(m.Ds[k][0], m.Ds[k][0]), D1 = pk(m.Ds[k][1], m.Ds[k][1]),
                         D2 = pk(m.Ds[k][2], m.Ds[k][2]);
                const f2 E0 = pk(-m.Ds[k][0], -m.Ds[k][0]), E1 = pk(-m.Ds[k][1], -m.Ds[k][1]),
                         E2 = pk(-m.Ds[k][2], -m.Ds[k][2]);
                h[0] = fma2(n[1], D2, fma2(n[2], E1, h[0]));
                h[1] = fma2(n[2], D0, fma2(n[0], E2, h[1]));
                h[2] = fma2(n[0], D1, fma2(n[1], E0, h[2]));
            }
        }
        return;
    }
    const f2 J = pk(m.J[kp], m.J[kp]);
#pragma unroll
    for (int c = 0; c < 3; ++c) h[c] = fma2(J, add2(P[c], M[c]), h[c]);
    if (DK == kDmiAxial) {   // Ds(+a) = D_a e_a
        const float D = A == 0 ? m.Ds[kp][A] * flip : m.Ds[kp][A];
        const f2 Dp = pk(D, D);
        constexpr int u = (A + 1) % 3, v = (A + 2) % 3;   // field (s x D e_A): h_u += D s_v, h_v -= D s_u
        const f2 du = sub2(M[u], P[u]), dv = sub2(P[v], M[v]);
        h[u] = fma2(Dp, dv, h[u]);
        h[v] = fma2(Dp, du, h[v]);
        if (EF) {
            d[u] = fma2(Dp, dv, d[u]);
            d[v] = fma2(Dp, du, d[v]);
        }
    } else {                 // (s+ - s-) x Ds(+a)
        const float f = A == 0 ? flip : 1.0f;
        const float D0 = m.Ds[kp][0] * f, D1 = m.Ds[kp][1] * f, D2 = m.Ds[kp][2] * f;
        const f2 dx = sub2(P[0], M[0]), dy = sub2(P[1], M[1]), dz = sub2(P[2], M[2]);
        h[0] = fma2(dy, pk(D2, D2), fma2(dz, pk(-D1, -D1), h[0]));
        h[1] = fma2(dz, pk(D0, D0), fma2(dx, pk(-D2, -D2), h[1]));
        h[2] = fma2(dx, pk(D1, D1), fma2(dy, pk(-D0, -D0), h[2]));
        if (EF) {
            d[0] = fma2(dy, pk(D2, D2), fma2(dz, pk(-D1, -D1), d[0]));
            d[1] = fma2(dz, pk(D0, D0), fma2(dx, pk(-D2, -D2), d[1]));
            d[2] = fma2(dx, pk(D1, D1), fma2(dy, pk(-D0, -D0), d[2]));
        }
    }
}

// Field (and DMI part) of a pair or a quad for one axis; x uses the same-row and shifted neighbours.
template <int DK, bool EF>
__device__ __forceinline__ void pair_axis_x(const DevModel& m, const f2 (&same)[3], const f2 (&sh)[3], bool xp,
                                            f2 (&h)[3], f2 (&d)[3]) {
    // xp = 1: +x is the shifted neighbour. The +-pair kinds fold the order into a sign.
    const float flip = 1.0f - 2.0f * (float)!xp;   // (sh - same) = flip * (s+ - s-)
    if (DK == kDmiPairs || DK == kDmiAxial) {
        axis_terms<DK, 0, EF>(m, sh, same, flip, h, d);
    } else {
        f2 P[3], M[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            P[c].v = xp ? sh[c].v : same[c].v;
            M[c].v = xp ? same[c].v : sh[c].v;
        }
        axis_terms<DK, 0, EF>(m, P, M, flip, h, d);
    }
}

template <int DK, bool EF>
__device__ __forceinline__ void quad_axis_x(const DevModel& m, const F2x2 (&same)[3], const F2x2 (&sh)[3], bool xp,
                                            f2 (&h)[2][3], f2 (&d)[2][3]) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        f2 a[3], b[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a[c] = j ? same[c].b : same[c].a;
            b[c] = j ? sh[c].b : sh[c].a;
        }
        pair_axis_x<DK, EF>(m, a, b, xp, h[j], d[j]);
    }
}

template <int DK, int A, bool EF>
__device__ __forceinline__ void quad_axis(const DevModel& m, const F2x2 (&up)[3], const F2x2 (&dn)[3],
                                          f2 (&h)[2][3], f2 (&d)[2][3]) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        f2 P[3], M[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            P[c] = j ? up[c].b : up[c].a;
            M[c] = j ? dn[c].b : dn[c].a;
        }
        axis_terms<DK, A, EF>(m, P, M, 1.0f, h[j], d[j]);
    }
}

// A pair of proposals (sphere_proposal) and the logarithms of their acceptance uniforms.
struct PairProp { f2 t[3], lu; };

__device__ __forceinline__ PairProp pair_propose(const nmmc_u4& r0, const nmmc_u4& r1) {
    const f2 c = pk(-0.99999994f, -0.99999994f), two = pk(2.0f, 2.0f), mone = pk(-1.0f, -1.0f);
    const f2 u0 = add2(pk(nmmc_u12f(r0.x), nmmc_u12f(r1.x)), c);
    const f2 u1 = add2(pk(nmmc_u12f(r0.y), nmmc_u12f(r1.y)), c);
    const f2 u2 = add2(pk(nmmc_u12f(r0.z), nmmc_u12f(r1.z)), c);
    PairProp p;
    p.t[2] = fma2(two, u0, mone);
    const f2 phi = mul2(fma2(two, u1, mone), pk(kPi, kPi));
    float sp0, cp0, sp1, cp1;
    __sincosf(lo(phi), &sp0, &cp0);
    __sincosf(hi(phi), &sp1, &cp1);
    const float z0 = lo(p.t[2]), z1 = hi(p.t[2]);
    const float w0 = fmaf(-z0, z0, 1.0f), w1 = fmaf(-z1, z1, 1.0f);
    const f2 rxy = mul2(pk(w0, w1), pk(rsqrt_norm(w0), rsqrt_norm(w1)));
    p.t[0] = mul2(rxy, pk(cp0, cp1));
    p.t[1] = mul2(rxy, pk(sp0, sp1));
    p.lu = mul2(pk(log2_norm(lo(u2)), log2_norm(hi(u2))), pk(kLn2, kLn2));
    return p;
}

// Metropolis tests of a pair of sites (heis_accept for each half): s becomes the new spins; true
// when either site accepted.
__device__ __forceinline__ bool pair_accept(const f2 (&h)[3], f2 (&s)[3], float beta, const PairProp& p) {
    const f2 dx = sub2(s[0], p.t[0]), dy = sub2(s[1], p.t[1]), dz = sub2(s[2], p.t[2]);
    const f2 dE = fma2(h[2], dz, fma2(h[1], dy, mul2(h[0], dx)));
    const f2 q = mul2(dE, pk(-beta, -beta));
    const bool a0 = (lo(dE) <= 0.0f) || (lo(q) > lo(p.lu));
    const bool a1 = (hi(dE) <= 0.0f) || (hi(q) > hi(p.lu));
#pragma unroll
    for (int c = 0; c < 3; ++c) s[c] = pk(a0 ? lo(p.t[c]) : lo(s[c]), a1 ? hi(p.t[c]) : hi(s[c]));
    return a0 | a1;
}

__device__ __forceinline__ bool pair_try(const f2 (&h)[3], f2 (&s)[3], float beta, const nmmc_u4& r0,
                                         const nmmc_u4& r1) {
    return pair_accept(h, s, beta, pair_propose(r0, r1));
}

}  // namespace nmmc
