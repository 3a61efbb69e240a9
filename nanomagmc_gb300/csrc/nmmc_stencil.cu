// Shared-memory resident sweeps of unmasked Heisenberg lattices in their stencil layout, one
// chain per thread-block cluster.
//
// The record kernel (nmmc_resident.cu) keeps only filled sites and gives each one a record of
// neighbour indices, so that Weibull particles of any size pack densely. An unmasked lattice
// needs no records: a cluster of C CTAs (1 to 16) holds one chain, cut into slabs of whole rows
// (2-D) or whole planes (3-D), and every thread updates four consecutive same-colour sites of a
// row with the packed arithmetic of nmmc_quad.cuh. Each CTA also keeps a copy of the row or
// plane below and above its slab; a thread that accepts a move in a boundary row stores it into
// the neighbour CTA's copy through distributed shared memory, and one cluster barrier per
// half-sweep orders the colours. The spins leave shared memory once per call.
//
// What bounds it: with many chains (C = 1, several CTAs per SM) instruction issue, as the
// streaming half-sweep; with few chains the latency of one update chain plus the barrier, so
// the next half-sweep's draws and proposals are computed between the barrier's arrive and wait.
// The streaming path pays a launch of about 4.8 us per half-sweep there.
//
// Layout in shared memory: [colour][slab unit, with the two copies][row][quad][component][4]
// floats. The three components of a quad lie 16 bytes apart, so a neighbour row costs one
// address; 48-byte steps between the lanes of a 16-byte access hit different banks. Rows that
// are not a multiple of four sites per colour end in a quad with padding: on periodic lattices
// the first padding element repeats the row's first site, which makes it the +x neighbour of the
// last one. Open edges read zeros (empty copies, padding and one zero quad), which add nothing.
//
// The per-site arithmetic, the draws and their counters are those of the streaming kernels, so
// every path gives the same chain bit for bit. With MEASURE the observables are computed from
// the spins still in shared memory after the last sweep: FP32 per thread and warp, FP64 across
// warps and CTAs in a fixed order, finished by one warp per chain.
#include <algorithm>

#include "nmmc_quad.cuh"

namespace nmmc {

namespace {

constexpr int kStThreads = 768;     // 80 registers: 24 warps per SM in one, two or three CTAs
constexpr int kStMaxCluster = 16;
constexpr int kQuadBytes = 48;

struct StencilArgs {
    float* spins;
    const float4* bh;
    unsigned long long* sweep;
    const int* chains;
    int nsweeps;
    int C;                   // CTAs per chain
    int NU, R, U;            // slab units of the lattice, rows per unit, largest slab
    int qpr, ipr;            // quads and thread items per row (rounded up)
    FastDiv div_ipr, div_pairs, div_rows, div_cols;   // items, pairs, rows per unit; load columns
    const double* Hd;
    double* obs;
    double* q;               // nullptr: not wanted
    double* acc;
    int nslices, accumulate;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The address of this CTA's shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(const void* p, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_st(uint32_t a, f2 v) {
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v.v) : "memory");
}
__device__ __forceinline__ void peer_st(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void peer_st(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ F2x2 lds_quad(const char* p, int c) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p + 16 * c);
    return F2x2{{t.x}, {t.y}};
}
}  // namespace

// One item is NP pairs of sites: a quad (NP = 2) where the chains fill the GPU, a pair (NP = 1)
// where they leave it short of warps.
template <int DIM, int DK, int NP, bool MEASURE>
__global__ void __launch_bounds__(kStThreads, 1) k_resident_stencil(const DevModel m, const StencilArgs g) {
    extern __shared__ __align__(16) char st_sm[];
    __shared__ float wred[kStThreads / 32][kNP];
    __shared__ double cred[kStMaxCluster][kNP];   // rank 0: the CTAs' totals
    const int C = g.C, rank = C > 1 ? (int)cluster_rank() : 0;
    const int ci = blockIdx.x / C, chain = g.chains[ci];
    const int tid = threadIdx.x;
    const bool per = m.periodic;
    const int hx = m.hx, qpr = g.qpr, ipr = g.ipr, R = g.R, NU = g.NU;
    const int u0 = rank * NU / C, nu = (rank + 1) * NU / C - u0;
    const int rowb = qpr * kQuadBytes, unitb = R * rowb, colb = (g.U + 2) * unitb;
    char* const zero = st_sm;                       // one quad of zeros
    char* const base = st_sm + kQuadBytes;          // colour 0, then colour 1
    // the slabs below and above: their CTA and where in its copies this slab's edge units go
    const int lo_rank = rank > 0 ? rank - 1 : C - 1, hi_rank = rank + 1 < C ? rank + 1 : 0;
    const bool has_lo = per || rank > 0, has_hi = per || rank + 1 < C;
    const int lo_slot = (lo_rank + 1) * NU / C - lo_rank * NU / C + 1;   // past its last unit
    const size_t P = (size_t)m.nhalf_pad;
    float* const gsp = g.spins + (size_t)chain * 6 * P;

    // a periodic lattice of whole quads overwrites every site of the slab and its copies
    const bool whole = (hx & 3) == 0;
    for (int i = tid; i < (whole && per ? kQuadBytes : kQuadBytes + 2 * colb) / 16; i += blockDim.x)
        reinterpret_cast<float4*>(st_sm)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // units u0 - 1 .. u0 + nu: the slab and its two copies. The rows of a plane are contiguous over
    // the units, so a place in the slab is decoded once for the six planes (three components of
    // two colours), whose loads are in flight together. With three divisions per site and plane
    // 8 chains of 30^3 took 8 us to load; with this, the same for the stores and the sums at the end,
    // a call of 10 sweeps with observables went from 70 to 59 us.
    const int ncol = whole ? qpr : hx + 1;   // float4 columns, or sites and the padding repeat
    {
        const int total = (nu + 2) * R * ncol, all = NU * R, first = (u0 - 1) * R;
#pragma unroll 2
        for (int i = tid; i < total; i += blockDim.x) {
            const int r = fdiv(i, g.div_cols), h = i - r * ncol;
            int gr = first + r;   // row of the lattice
            if (gr < 0 || gr >= all) {
                if (!per) continue;
                gr += gr < 0 ? all : -all;
            }
            if (whole) {
                const float4* src = reinterpret_cast<const float4*>(gsp + (size_t)gr * hx) + h;
                float4* dst = reinterpret_cast<float4*>(base + r * rowb + h * kQuadBytes);
                float4 v[6];
#pragma unroll
                for (int pl = 0; pl < 6; ++pl) v[pl] = __ldg(src + pl * (P / 4));
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    dst[c] = v[c];
                    dst[colb / 16 + c] = v[3 + c];
                }
            } else if (h < hx || per) {
                const float* src = gsp + (size_t)gr * hx + (h < hx ? h : 0);
                char* dst = base + r * rowb + (h >> 2) * kQuadBytes + 4 * (h & 3);
                float v[6];
#pragma unroll
                for (int pl = 0; pl < 6; ++pl) v[pl] = __ldg(src + pl * P);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    *reinterpret_cast<float*>(dst + 16 * c) = v[c];
                    *reinterpret_cast<float*>(dst + colb + 16 * c) = v[3 + c];
                }
            }
        }
    }
    if (C > 1) {
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }

    const float4 p = g.bh[chain];
    const unsigned long long sw0 = g.sweep[chain];
    const int items = nu * R * ipr;

    // item `it` of the slab: its row r (unit r / R), row y of the unit, plane z, first site h0
    auto decode = [&](int it, int& r, int& h0, int& y, int& z) {
        r = fdiv(it, g.div_ipr);
        h0 = (it - r * ipr) * 2 * NP;
        if (DIM == 3) {
            const int ul = fdiv(r, g.div_rows);
            y = r - ul * R;
            z = u0 + ul;
        } else {
            y = u0 + r;
            z = 0;
        }
    };
    auto propose = [&](int colour, int h0, int y, int z, unsigned long long sw, PairProp (&pp)[NP]) {
        const int xp = (y + z + colour) & 1;
        const uint32_t box = (uint32_t)(m.edge * (y + m.edge * z) + 2 * h0 + xp);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const nmmc_u4 ra = sweep_draw<true>(m, box + 4 * j, sw, (uint32_t)chain);
            const nmmc_u4 rb = sweep_draw<true>(m, box + 4 * j + 2, sw, (uint32_t)chain);
            pp[j] = pair_propose(ra, rb);
        }
    };
    // sites: a row's bytes are [quad][component][4 sites]
    auto site_at = [&](int h) { return (h >> 2) * kQuadBytes + (h & 3) * 4; };
    // the item's sites in the rows y -+ 1 (2-D: the units -+ 1, copies included)
    auto up_row = [&](const char* q, int y) -> const char* {
        if (DIM == 2) return q + unitb;
        return y + 1 < R ? q + rowb : (per ? q - (R - 1) * rowb : zero);
    };
    auto dn_row = [&](const char* q, int y) -> const char* {
        if (DIM == 2) return q - unitb;
        return y > 0 ? q - rowb : (per ? q + (R - 1) * rowb : zero);
    };
    // the x-neighbour outside the item whose first site h0 lies at q, in the row at `row`: site
    // h0 - 1 (xp = 0) or h0 + 2 NP. In a padded row the padding repeat stands for site hx.
    const int last = site_at(hx - 1);
    auto ex_site = [&](const char* row, const char* q, int h0, int xp) -> const char* {
        if (xp) {
            if (h0 + 2 * NP >= hx && (whole || NP == 2)) return per && whole ? row : zero;
            return NP == 2 ? q + kQuadBytes : q + ((h0 & 2) ? kQuadBytes - 8 : 8);
        }
        if (h0 == 0) return per ? row + last : zero;
        return NP == 2 || !(h0 & 2) ? q - kQuadBytes + 12 : q - 4;
    };
    auto lds_pair = [&](const char* q, int j, int c) -> f2 {
        return f2{*reinterpret_cast<const unsigned long long*>(q + 16 * c + 8 * j)};
    };

    PairProp pp[NP];
    int r1 = 0, h1 = 0, y1 = 0, z1 = 0;   // this thread's first item: the same in every half-sweep
    const bool mine = tid < items;
    // with pairs (few warps) the first item's proposals are ready before the barrier; with quads the
    // registers are worth more (420 chains of 64^2: 9.8 -> 9.5 us per sweep without)
    constexpr bool ahead = NP == 1;
    if (mine) {
        decode(tid, r1, h1, y1, z1);
        if (ahead && g.nsweeps > 0) propose(0, h1, y1, z1, sw0, pp);
    }
    for (int hs = 0; hs < 2 * g.nsweeps; ++hs) {
        const int colour = hs & 1;
        const unsigned long long sw = sw0 + (unsigned)(hs >> 1);
        char* const cown = base + colour * colb + unitb;          // unit 1: the slab's first
        const char* const coth = base + (colour ^ 1) * colb + unitb;
        int r = r1, h0 = h1, y = y1, z = z1;
        for (int it = tid; it < items; it += blockDim.x) {
            if (it != tid) decode(it, r, h0, y, z);
            if (it != tid || !ahead) propose(colour, h0, y, z, sw, pp);
            const int xp = (y + z + colour) & 1;
            const int at = site_at(h0);
            char* const own = cown + r * rowb + at;
            const char* const orow = coth + r * rowb;
            const char* const oth = orow + at;
            const char* const yu = up_row(oth, y);
            const char* const yd = dn_row(oth, y);
            const char* const exq = ex_site(orow, oth, h0, xp);
            f2 s[NP][3], h[NP][3], d[3];
            {
                f2 same[NP][3], sh[NP][3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float ex = *reinterpret_cast<const float*>(exq + 16 * c);
                    if (NP == 2) {
                        const F2x2 t = lds_quad(own, c), o = lds_quad(oth, c), q = shifted_quad(o, ex, xp != 0);
                        s[0][c] = t.a;
                        s[NP - 1][c] = t.b;
                        same[0][c] = o.a;
                        same[NP - 1][c] = o.b;
                        sh[0][c] = q.a;
                        sh[NP - 1][c] = q.b;
                    } else {
                        s[0][c] = lds_pair(own, 0, c);
                        const f2 o = lds_pair(oth, 0, c);
                        same[0][c] = o;
                        sh[0][c] = pk(xp ? hi(o) : ex, xp ? ex : lo(o));
                    }
                }
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    h[j][0] = pk(p.y, p.y);
                    h[j][1] = pk(p.z, p.z);
                    h[j][2] = pk(p.w, p.w);
                    pair_axis_x<DK, false>(m, same[j], sh[j], xp != 0, h[j], d);
                }
            }
#pragma unroll
            for (int ax = 1; ax < DIM; ++ax) {
                const char* const ua = ax == 1 ? yu : oth + unitb;
                const char* const da = ax == 1 ? yd : oth - unitb;
                f2 a[NP][3], b[NP][3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    if (NP == 2) {
                        const F2x2 t = lds_quad(ua, c), u = lds_quad(da, c);
                        a[0][c] = t.a;
                        a[NP - 1][c] = t.b;
                        b[0][c] = u.a;
                        b[NP - 1][c] = u.b;
                    } else {
                        a[0][c] = lds_pair(ua, 0, c);
                        b[0][c] = lds_pair(da, 0, c);
                    }
                }
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    if (ax == 1) axis_terms<DK, 1, false>(m, a[j], b[j], 1.0f, h[j], d);
                    else axis_terms<DK, 2, false>(m, a[j], b[j], 1.0f, h[j], d);
                }
            }
            bool any = false;
#pragma unroll
            for (int j = 0; j < NP; ++j) any |= pair_accept(h[j], s[j], p.x, pp[j]);
            if (any) {
                const int ul = DIM == 3 ? z - u0 : r;
                const bool to_lo = ul == 0 && has_lo, to_hi = ul == nu - 1 && has_hi;
                const int row_in_unit = DIM == 3 ? y * rowb : 0;
                char* const lo_row = base + colour * colb + lo_slot * unitb + row_in_unit;   // in CTA lo_rank
                char* const hi_row = base + colour * colb + row_in_unit;                     // in CTA hi_rank
                const int n = hx - h0;   // sites of the row from this item on
                const bool full = n >= 2 * NP;
                if (full) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if (NP == 2)
                            *reinterpret_cast<ulonglong2*>(own + 16 * c) = make_ulonglong2(s[0][c].v, s[NP - 1][c].v);
                        else
                            *reinterpret_cast<unsigned long long*>(own + 16 * c) = s[0][c].v;
                    }
                    if (to_lo) {
                        const uint32_t a = peer_addr(lo_row + at, lo_rank);
#pragma unroll
                        for (int c = 0; c < 3; ++c)
#pragma unroll
                            for (int j = 0; j < NP; ++j) peer_st(a + 16 * c + 8 * j, s[j][c]);
                    }
                    if (to_hi) {
                        const uint32_t a = peer_addr(hi_row + at, hi_rank);
#pragma unroll
                        for (int c = 0; c < 3; ++c)
#pragma unroll
                            for (int j = 0; j < NP; ++j) peer_st(a + 16 * c + 8 * j, s[j][c]);
                    }
                }
                if (!whole && (!full || (h0 == 0 && per))) {
                    // a part-filled item stores its sites one by one; a row's first item also the
                    // padding repeat of its first site
                    const uint32_t la = peer_addr(lo_row, lo_rank), ha = peer_addr(hi_row, hi_rank);
                    const int pad = site_at(hx);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
#pragma unroll
                        for (int k = 0; k < 2 * NP - 1; ++k) {
                            if (full || k >= n) continue;
                            const float v = (k & 1) ? hi(s[k >> 1][c]) : lo(s[k >> 1][c]);
                            *reinterpret_cast<float*>(own + 16 * c + 4 * k) = v;
                            if (to_lo) peer_st(la + at + 16 * c + 4 * k, v);
                            if (to_hi) peer_st(ha + at + 16 * c + 4 * k, v);
                        }
                        if (h0 == 0 && per) {
                            *reinterpret_cast<float*>(own + pad + 16 * c) = lo(s[0][c]);
                            if (to_lo) peer_st(la + pad + 16 * c, lo(s[0][c]));
                            if (to_hi) peer_st(ha + pad + 16 * c, lo(s[0][c]));
                        }
                    }
                }
            }
        }
        // the next half-sweep's draws and proposals do not depend on spins: computed while the
        // other CTAs arrive
        const int nh = hs + 1;
        const bool more = mine && nh < 2 * g.nsweeps;
        if (C > 1) {
            cluster_arrive();
            if (more) propose(nh & 1, h1, y1, z1, sw0 + (unsigned)(nh >> 1), pp);
            cluster_wait();
        } else {
            if (more && ahead) propose(nh & 1, h1, y1, z1, sw0 + (unsigned)(nh >> 1), pp);
            __syncthreads();
        }
    }
    if constexpr (MEASURE) {
        // the streaming measurement kernel's per-site terms (Old/lib/thermodynamics.cpp:71-221)
        // over both colours of the slab; the angles are summed per plane in 3-D (a slice's charge)
        const int lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
        const bool pq = per && m.periodic_q;
        const int e4 = m.edge - m.edge % 4;
        // items of two sites (few registers), 32 items of one plane to a warp at a time
        const int pairs = (hx + 1) >> 1;
        const int grows = DIM == 3 ? R : nu * R, gitems = grows * pairs, ngroup = DIM == 3 ? nu : 1;
        const int chunks = (2 * gitems + 31) >> 5;
        float* const qpart = reinterpret_cast<float*>(base + 2 * colb);   // [plane][warp] angle sums
        for (int k = tid; k < ngroup * nw; k += blockDim.x) qpart[k] = 0.0f;
        float a[kNP];
#pragma unroll
        for (int k = 0; k < kNP; ++k) a[k] = 0.0f;
        __syncthreads();
        for (int ch = warp; ch < ngroup * chunks; ch += nw) {
            const int gr = ch / chunks, i2 = (ch - gr * chunks) * 32 + lane;
            a[10] = 0.0f;
            if (i2 < 2 * gitems) {
                const int colour = i2 >= gitems, it = i2 - colour * gitems;
                const int rg = fdiv(it, g.div_pairs), h0 = (it - rg * pairs) * 2;
                const int r = gr * grows + rg;
                const int y = DIM == 3 ? rg : u0 + rg, z = DIM == 3 ? u0 + gr : 0;
                const int xp = (y + z + colour) & 1, at = site_at(h0);
                const char* const own = base + colour * colb + unitb + r * rowb + at;
                const char* const orow = base + (colour ^ 1) * colb + unitb + r * rowb;
                const char* const oth = orow + at;
                const char* const yu = up_row(oth, y);
                const char* const yd = dn_row(oth, y);
                // the x-neighbour outside the pair
                int he = xp ? h0 + 2 : h0 - 1;
                if (he < 0) he = per ? hx - 1 : -1;
                else if (he >= hx) he = whole ? (per ? 0 : -1) : (he == hx ? hx : -1);
                const char* const exq = he < 0 ? zero : orow + site_at(he);
                float sv[3][2], n[3][2 * DIM][2];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    auto two = [&](const char* q, float (&o)[2]) {
                        const float2 t = *reinterpret_cast<const float2*>(q + 16 * c);
                        o[0] = t.x;
                        o[1] = t.y;
                    };
                    float same[2];
                    two(own, sv[c]);
                    two(oth, same);
                    const float ex = *reinterpret_cast<const float*>(exq + 16 * c);
                    const float sh[2] = {xp ? same[1] : ex, xp ? ex : same[0]};
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        n[c][0][k] = xp ? sh[k] : same[k];
                        n[c][1][k] = xp ? same[k] : sh[k];
                    }
                    two(yu, n[c][2]);
                    two(yd, n[c][3]);
                    if (DIM == 3) {
                        two(oth + unitb, n[c][2 * DIM - 2]);
                        two(oth - unitb, n[c][2 * DIM - 1]);
                    }
                }
                const bool qyu = y + 1 < m.edge || pq, qyd = y >= 1 || pq;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (h0 + k >= hx) continue;
                    const int x = 2 * (h0 + k) + xp;
                    const float s0 = sv[0][k], s1 = sv[1][k], s2 = sv[2][k];
                    float f0 = 0.f, f1 = 0.f, f2v = 0.f;
#pragma unroll
                    for (int ax = 0; ax < DIM; ++ax) {
                        const int kp = 2 * ax, km = 2 * ax + 1;
                        const float a0 = n[0][kp][k], a1 = n[1][kp][k], a2 = n[2][kp][k];
                        const float b0 = n[0][km][k], b1 = n[1][km][k], b2 = n[2][km][k];
                        if (DK <= kDmiGeneral) {
                            f0 = fmaf(m.J[km], b0, fmaf(m.J[kp], a0, f0));
                            f1 = fmaf(m.J[km], b1, fmaf(m.J[kp], a1, f1));
                            f2v = fmaf(m.J[km], b2, fmaf(m.J[kp], a2, f2v));
                            if (DK == kDmiGeneral) {
                                f0 = fmaf(m.De[kp][1], a2, fmaf(-m.De[kp][2], a1, f0));
                                f1 = fmaf(m.De[kp][2], a0, fmaf(-m.De[kp][0], a2, f1));
                                f2v = fmaf(m.De[kp][0], a1, fmaf(-m.De[kp][1], a0, f2v));
                                f0 = fmaf(m.De[km][1], b2, fmaf(-m.De[km][2], b1, f0));
                                f1 = fmaf(m.De[km][2], b0, fmaf(-m.De[km][0], b2, f1));
                                f2v = fmaf(m.De[km][0], b1, fmaf(-m.De[km][1], b0, f2v));
                            }
                        } else {   // +-axis pairs: J (n+ + n-) + De(+a) x (n+ - n-)
                            const float J = m.J[kp], D0 = m.De[kp][0], D1 = m.De[kp][1], D2 = m.De[kp][2];
                            const float d0 = a0 - b0, d1 = a1 - b1, d2 = a2 - b2;
                            f0 = fmaf(J, a0 + b0, f0);
                            f1 = fmaf(J, a1 + b1, f1);
                            f2v = fmaf(J, a2 + b2, f2v);
                            if (DK == kDmiPairs || ax != 0) {
                                f0 = fmaf(D1, d2, fmaf(-D2, d1, f0));
                            }
                            if (DK == kDmiPairs || ax != 1) {
                                f1 = fmaf(D2, d0, fmaf(-D0, d2, f1));
                            }
                            if (DK == kDmiPairs || ax != 2) {
                                f2v = fmaf(D0, d1, fmaf(-D1, d0, f2v));
                            }
                        }
                    }
                    a[0] = fmaf(s0, f0, fmaf(s1, f1, fmaf(s2, f2v, a[0])));
                    a[1] += s0;
                    a[2] += s1;
                    a[3] += s2;
                    if (colour == 0) {   // subM(0): (sum of coordinates) % 2 == 0
                        a[4] += s0;
                        a[5] += s1;
                        a[6] += s2;
                    }
                    const int possum = x + y, posdiff = y - x + e4;   // C truncating remainders
                    const int z4 = z & 3;
                    if ((z4 & 1) == 0 && (possum & 3) == z4 && posdiff % 4 == z4) {
                        a[7] += s0;
                        a[8] += s1;
                        a[9] += s2;
                    }
                    const bool qxm = x >= 1 || pq, qxp = x + 1 < m.edge || pq;
                    if (qxm && qyu)
                        a[10] += solid_angle_f(s0, s1, s2, n[0][1][k], n[1][1][k], n[2][1][k], n[0][2][k],
                                               n[1][2][k], n[2][2][k]);
                    if (qxp && qyd)
                        a[10] += solid_angle_f(s0, s1, s2, n[0][0][k], n[1][0][k], n[2][0][k], n[0][3][k],
                                               n[1][3][k], n[2][3][k]);
                }
            }
            float v = a[10];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) qpart[gr * nw + warp] += v;   // this warp's own slot
        }
#pragma unroll
        for (int k = 0; k < kNP - 1; ++k) {
            float v = a[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) wred[warp][k] = v;
        }
        __syncthreads();
        // FP64 sums over the warps, side by side (an FP64 addition takes about 40 cycles here, so one
        // warp adding up 24 warps' totals and angles took 5 us): a tree per total in the warps
        // 0-9, the angles in the warp after them (the last one, where there are fewer)
        auto put = [&](int k, double v) {
            if (rank == 0) cred[0][k] = v;
            else peer_st(peer_addr(&cred[rank][k], 0), v);
        };
        for (int k = warp; k < kNP - 1; k += nw) {
            double v = lane < nw ? (double)wred[lane][k] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) put(k, v);
        }
        if (warp == (nw > kNP - 1 ? kNP - 1 : nw - 1)) {
            double qsum = 0.0;
            if (DIM == 2) {
                qsum = lane < nw ? (double)qpart[lane] : 0.0;
            } else {   // a lane per plane: the slice's charge
                for (int gr = lane; gr < ngroup; gr += 32) {
                    double t0 = 0.0, t1 = 0.0;
                    for (int w = 0; w + 1 < nw; w += 2) {
                        t0 += (double)qpart[gr * nw + w];
                        t1 += (double)qpart[gr * nw + w + 1];
                    }
                    if (nw & 1) t0 += (double)qpart[gr * nw + nw - 1];
                    t0 += t1;
                    qsum += t0;
                    if (g.q) g.q[(size_t)ci * g.nslices + u0 + gr] = t0 / (2 * M_PI);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) qsum += __shfl_down_sync(0xffffffffu, qsum, o);
            if (lane == 0) put(kNP - 1, qsum);
        }
        if (C > 1) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
        if (rank == 0 && warp == 0) {
            double v = 0.0;
            if (lane < kNP)
                for (int k = 0; k < C; ++k) v += cred[k][lane];
            const double qv = __shfl_sync(0xffffffffu, v, kNP - 1) / (2 * M_PI);
            if (DIM == 2 && g.q && lane == 0) g.q[ci] = qv;
            finalize_chain_warp(v, lane, g.Hd + 3 * (size_t)chain, qv, g.obs + (size_t)ci * NMMC_OBS_N,
                                g.acc + (size_t)chain * NMMC_ACC_N, g.accumulate);
        }
    }
    // the slab back to HBM, without its copies
    {
        const int total = nu * R * ncol;   // the places of the load (a padding repeat is left out)
#pragma unroll 2
        for (int i = tid; i < total; i += blockDim.x) {
            const int r = fdiv(i, g.div_cols), h = i - r * ncol;
            float* dst = gsp + (size_t)(u0 * R + r) * hx;
            const char* src = base + unitb + r * rowb;
            if (whole) {
                const float4* q = reinterpret_cast<const float4*>(src + h * kQuadBytes);
#pragma unroll
                for (int pl = 0; pl < 6; ++pl)
                    reinterpret_cast<float4*>(dst + pl * P)[h] = q[(pl >= 3 ? colb / 16 : 0) + pl % 3];
            } else if (h < hx) {
                const char* q = src + site_at(h);
#pragma unroll
                for (int pl = 0; pl < 6; ++pl)
                    dst[pl * P + h] = *reinterpret_cast<const float*>(q + (pl >= 3 ? colb : 0) + 16 * (pl % 3));
            }
        }
    }
    if (rank == 0 && tid == 0) g.sweep[chain] = sw0 + (unsigned long long)g.nsweeps;
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
namespace {

using StencilFn = void (*)(const DevModel, const StencilArgs);

template <int DIM, int NP, bool MEASURE>
StencilFn stencil_kernel_dk(int dk) {
    switch (dk) {
        case kDmiNone: return k_resident_stencil<DIM, kDmiNone, NP, MEASURE>;
        case kDmiGeneral: return k_resident_stencil<DIM, kDmiGeneral, NP, MEASURE>;
        case kDmiPairs: return k_resident_stencil<DIM, kDmiPairs, NP, MEASURE>;
        default: return k_resident_stencil<DIM, kDmiAxial, NP, MEASURE>;
    }
}

template <int DIM, bool MEASURE>
StencilFn stencil_kernel_np(int dk, int np) {
    return np == 1 ? stencil_kernel_dk<DIM, 1, MEASURE>(dk) : stencil_kernel_dk<DIM, 2, MEASURE>(dk);
}

StencilFn stencil_kernel(const Ctx& c, int np, bool measure) {
    const int dk = c.m.dmi_kind;
    if (c.dim == 3) return measure ? stencil_kernel_np<3, true>(dk, np) : stencil_kernel_np<3, false>(dk, np);
    return measure ? stencil_kernel_np<2, true>(dk, np) : stencil_kernel_np<2, false>(dk, np);
}

int units_of(const Ctx& c) { return c.dim == 3 ? c.m.lz : c.m.ly; }
int rows_of(const Ctx& c) { return c.dim == 3 ? c.m.ly : 1; }
int quads_per_row(const Ctx& c) { return (c.m.hx + 3) / 4; }

// Dynamic shared memory of a CTA with 1/C of a chain.
size_t stencil_bytes(const Ctx& c, int C) {
    const size_t U = (units_of(c) + C - 1) / C;
    return kQuadBytes + 2 * (U + 2) * (size_t)rows_of(c) * quads_per_row(c) * kQuadBytes +
           (c.dim == 3 ? U : 1) * (kStThreads / 32) * sizeof(float);   // with the planes' angle sums
}

size_t stencil_budget(const Ctx& c) {
    const size_t fixed = sizeof(float) * (kStThreads / 32) * kNP + sizeof(double) * kStMaxCluster * kNP + 64;
    return c.smem_optin > fixed ? c.smem_optin - fixed : 0;
}

cudaLaunchConfig_t stencil_config(int n, const StencilShape& s, cudaStream_t stream, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)n * s.C);
    cfg.blockDim = dim3(s.threads);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = stream;
    if (s.C > 1) {
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = s.C;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cfg;
}

// Both limits are raised to this device's maximum, the same value in every context: a kernel's
// attributes belong to the process, so a context that set only what it needs would lower them
// for the others.
int stencil_attrs(const Ctx& c) {
    for (int v = 0; v < 4; ++v) {
        const void* k = (const void*)stencil_kernel(c, 1 + (v & 1), v >= 2);
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stencil_budget(c));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return cuda_check(e, "stencil kernel attributes");
    }
    return NMMC_OK;
}

// Items of a CTA's largest slab with np pairs per item.
int stencil_items(const Ctx& c, int C, int np) {
    const int U = (units_of(c) + C - 1) / C;
    return U * rows_of(c) * ((c.m.hx + 2 * np - 1) / (2 * np));
}

// Item size and threads of a CTA. 768 threads per SM (the register file at 80 each) are shared by
// the CTAs that run on one; quads, unless pairs still leave every thread at most one item.
void stencil_width(const Ctx& c, int n, StencilShape& s) {
    const size_t fit = std::max<size_t>(1, (c.smem_optin + 1024) / (s.smem + 4096));
    const int share = (int)std::min<size_t>(std::min(fit, (size_t)3), (size_t)((long)n * s.C + c.sm_count - 1) / c.sm_count);
    const int most = kStThreads / std::max(1, share) / 32 * 32;
    s.np = stencil_items(c, s.C, 1) <= most ? 1 : 2;
    const int items = stencil_items(c, s.C, s.np), each = (items + most - 1) / most;
    s.threads = std::max(32, ((items + each - 1) / each + 31) / 32 * 32);
}

// Clusters of C CTAs that run at the same time (0: none fits).
int active_clusters(const Ctx& c, const StencilShape& s) {
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = stencil_config(1, s, c.stream, &at);
    int k = 0;
    const void* f = (const void*)stencil_kernel(c, s.np, true);   // the variant with the larger footprint
    cudaError_t e;
    if (s.C > 1) {
        e = cudaOccupancyMaxActiveClusters(&k, f, &cfg);
    } else {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, f, s.threads, s.smem);
        k *= c.sm_count;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return k;
}

}  // namespace

// The shape of a call on n chains (C = 0: the lattice is not covered, or does not fit). The time
// of a half-sweep is close to 1000 cycles (update latency and barrier) plus 2.2 cycles for every
// site that the CTAs sharing an SM update, once per wave of clusters that run together; C is the
// smallest cluster with the least of that. Measured per sweep, model against time at 1.92 GHz:
// 16 chains of 128^2 C = 16 3.4 / 3.3 us, C = 8 (two waves) 6.8 / 5.0; 8 of 30^3 C = 10 4.3 / 4.6,
// C = 8 5.4 / 6.1, C = 16 (two waves) 5.4 / 6.9; 420 of 64^2 C = 1 15 / 9.6, C = 2 26 / 9.9 (two
// waves overlap there, but do not win).
StencilShape stencil_shape(const Ctx& c, int n) {
    StencilShape best;
    if (c.ising || c.masked || c.m.general || n <= 0 || stencil_attrs(c) != NMMC_OK) return best;
    double best_cost = 0;
    for (int C = 1; C <= kStMaxCluster && C <= units_of(c); ++C) {
        StencilShape s;
        s.C = C;
        s.smem = stencil_bytes(c, C);
        if (s.smem > stencil_budget(c) || s.smem / 4 > 65535) continue;   // 65535: FastDiv's range
        stencil_width(c, n, s);
        auto cost_of = [&](int active) {
            const int waves = (n + active - 1) / active, at_once = std::min(n, active);
            const int per_sm = (int)(((long)at_once * C + c.sm_count - 1) / c.sm_count);
            return waves * (1000.0 + 2.2 * per_sm * stencil_items(c, C, s.np) * 2 * s.np);
        };
        if (best.C && cost_of(n) >= 0.99 * best_cost) continue;   // not even with every cluster running
        const int active = active_clusters(c, s);
        if (active < 1) continue;
        const double cost = cost_of(active);
        if (!best.C || cost < 0.99 * best_cost) {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

// nsweeps sweeps of the listed chains (d_chains, n entries, each chain at most once) and, with
// measure, their observables in list order and (accumulate) their accumulators.
int launch_stencil_sweeps(Ctx& c, const int* d_chains, int n, int nsweeps, bool measure, int accumulate) {
    if (n <= 0) return NMMC_OK;
    auto known = c.st_shapes.find(n);
    if (known == c.st_shapes.end()) known = c.st_shapes.emplace(n, stencil_shape(c, n)).first;
    const StencilShape& s = known->second;
    if (s.C < 1) return set_error(NMMC_ERR_UNSUPPORTED, "lattice does not fit the stencil resident kernel");
    StencilArgs g{};
    g.spins = (float*)c.d_spins;
    g.bh = c.d_bh;
    g.sweep = c.d_sweep;
    g.chains = d_chains;
    g.nsweeps = nsweeps;
    g.C = s.C;
    g.NU = units_of(c);
    g.R = rows_of(c);
    g.U = (g.NU + s.C - 1) / s.C;
    g.qpr = quads_per_row(c);
    g.ipr = (c.m.hx + 2 * s.np - 1) / (2 * s.np);
    g.div_ipr = fast_div(g.ipr);
    g.div_pairs = fast_div((c.m.hx + 1) / 2);
    g.div_rows = fast_div(g.R);
    g.div_cols = fast_div(c.m.hx % 4 ? c.m.hx + 1 : g.qpr);
    g.Hd = c.d_Hd;
    g.obs = c.d_obs;
    g.q = c.d_q;
    g.acc = c.d_acc;
    g.nslices = c.nslices;
    g.accumulate = accumulate;
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = stencil_config(n, s, c.stream, &at);
    return cuda_check(cudaLaunchKernelEx(&cfg, stencil_kernel(c, s.np, measure), (const DevModel)c.m, (const StencilArgs)g),
                      "k_resident_stencil");
}

}  // namespace nmmc
