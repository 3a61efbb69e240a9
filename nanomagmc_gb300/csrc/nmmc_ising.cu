// Streaming half-sweeps and observables of unmasked Ising lattices, four sites to a 32-bit word.
//
// Ising spins are one byte each (+1, -1), so a word holds four consecutive same-colour sites of a
// row. A site's Metropolis test depends only on the signs of its 2*dim neighbours and its own:
// k_ising_table turns the test "dE <= 0 or -dE beta > log(u)" into "k < K" for each of those
// 2^(2*dim+1) patterns of a chain, with k the 23-bit integer behind the uniform u. K is found by
// bisection with the test itself (the same FP32 field, dE and logf as ising_try; logf does not
// decrease over the 2^23 uniforms), so every decision, and with it the chain, is the same bit for
// bit. The half-sweep then costs a generator block and a table look-up per site. A colour of 24
// chains of 64^3 (3.1 M updates): 32.8 us for the one-site kernel with its float field and logf
// (ALU 59 %, issue 75 % busy), 13.9 us for the words (71 per
// update, the FMA-heavy pipe of the generator's multiplies 61 % busy); observables 65.6 -> 16.5 us.
#include "nmmc_kernels.cuh"

namespace nmmc {

namespace {

constexpr uint32_t kAllK = 1u << 23;     // every uniform accepts
constexpr int kItabMax = 128;            // 2^(2*3+1) patterns

// The four sites' neighbours (or own) signs into bit `bit` of each byte of the pattern word.
__device__ __forceinline__ uint32_t sign_bits(uint32_t w, int bit) { return (w >> (7 - bit)) & (0x01010101u << bit); }

// Words of an item's row piece: W words (4W sites) at byte offset `off` (4W-byte aligned).
template <int W>
struct Words { uint32_t w[W]; };
template <int W>
__device__ __forceinline__ Words<W> ld_words(const int8_t* p) {
    Words<W> r;
    if (W == 4) {
        const uint4 t = *reinterpret_cast<const uint4*>(p);
        r.w[0] = t.x;
        r.w[W > 1 ? 1 : 0] = t.y;
        r.w[W > 2 ? 2 : 0] = t.z;
        r.w[W > 3 ? 3 : 0] = t.w;
    } else {
        r.w[0] = *reinterpret_cast<const uint32_t*>(p);
    }
    return r;
}

// The x-neighbours that are not the same-index sites: compact indices + 1 (xp = 1) or - 1;
// `ex` is the byte outside the item.
template <int W>
__device__ __forceinline__ uint32_t shifted_word(const Words<W>& same, int i, uint32_t ex, int xp) {
    const uint32_t next = i + 1 < W ? same.w[i + 1 < W ? i + 1 : i] : ex;
    const uint32_t prev = i > 0 ? same.w[i > 0 ? i - 1 : 0] : ex << 24;
    return xp ? __byte_perm(same.w[i], next, 0x4321) : __byte_perm(prev, same.w[i], 0x6543);
}

}  // namespace

// One block of 128 threads per chain: entry e of its table, bit k of e the sign of neighbour k
// (1: -1), bit 2*dim the site's own.
__global__ void __launch_bounds__(kItabMax) k_ising_table(const DevModel m, const float4* __restrict__ bh,
                                                          uint32_t* __restrict__ tab) {
    const int nd = 2 * m.dim, e = threadIdx.x;
    if (e >= 2 << nd) return;
    const float4 p = bh[blockIdx.x];
    float h = p.y;
    for (int k = 0; k < nd; ++k) h = fmaf(m.J[k], (e >> k) & 1 ? -1.0f : 1.0f, h);
    const float so = (e >> nd) & 1 ? -1.0f : 1.0f;
    const float dE = h * (so - (-so));   // the proposal -so; the other one changes nothing
    uint32_t lo = 0, hi = kAllK;         // first k that rejects: in [lo, hi]
    if (dE <= 0.0f) {
        lo = kAllK;
    } else {
        const float x = -dE * p.x;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (x > logf(nmmc_u01f(mid << 9))) lo = mid + 1;
            else hi = mid;
        }
    }
    tab[(size_t)blockIdx.x * kItabMax + e] = lo;
}

// One colour of every listed chain; a thread updates 4W consecutive sites of a row.
template <int DIM, bool PERIODIC, int W>
__global__ void __launch_bounds__(256)
k_ising_words(const DevModel m, int8_t* spins, const float4* __restrict__ bh,
              const unsigned long long* sweep, const int* __restrict__ chains,
              const uint32_t* __restrict__ tab, int colour, unsigned sweep_off) {
    seq_begin();
    constexpr int ND = 2 * DIM;
    __shared__ uint32_t st[2 << ND];
    const int chain = chains[blockIdx.y];
    if (threadIdx.x < (2 << ND)) st[threadIdx.x] = tab[(size_t)chain * kItabMax + threadIdx.x];
    __syncthreads();
    const int ipr = m.hx / (4 * W);
    const int item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= ipr * m.ly * m.lz) return;
    const int row = item / ipr, h0 = (item - row * ipr) * 4 * W;
    const int z = DIM == 3 ? row / m.ly : 0, y = row - z * m.ly;
    const int xp = (y + z + colour) & 1;
    const size_t P = (size_t)m.nhalf_pad;
    int8_t* own = spins + ((size_t)chain * 2 + colour) * P;
    const int8_t* oth = spins + ((size_t)chain * 2 + (colour ^ 1)) * P;
    const int rb = row * m.hx + h0;
    const int hrow = row * m.hx;
    bool full = true;   // every site of the item has all its neighbours
    int ho = xp ? h0 + 4 * W : h0 - 1, yu = y + 1, yd = y - 1, zu = z + 1, zd = z - 1;
    if (PERIODIC) {
        ho = ho < 0 ? m.hx - 1 : (ho >= m.hx ? 0 : ho);
        yu = yu == m.ly ? 0 : yu;
        yd = yd < 0 ? m.ly - 1 : yd;
        zu = zu == m.lz ? 0 : zu;
        zd = zd < 0 ? m.lz - 1 : zd;
    } else {
        full = ho >= 0 && ho < m.hx && yu < m.ly && yd >= 0 && (DIM == 2 || (zu < m.lz && zd >= 0));
    }
    const unsigned long long sw = sweep[chain] + sweep_off;
    const uint32_t box = (uint32_t)(m.edge * (y + m.edge * z) + 2 * h0 + xp);
    if (!PERIODIC && !full) {
        // at an open edge: the one-site arithmetic, absent neighbours reading 0
        const float4 p = bh[chain];
#pragma unroll 1
        for (int k = 0; k < 4 * W; ++k) {
            float n[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const int j = nb_compact<false>(m, 2 * (h0 + k) + xp, y, z, d);
                n[d] = j >= 0 ? (float)oth[j] : 0.0f;
            }
            const nmmc_u4 r = sweep_draw<true>(m, box + 2 * k, sw, (uint32_t)chain);
            float t;
            if (ising_attempt<ND>(m, (float)own[rb + k], n, p, r, t)) own[rb + k] = (int8_t)t;
        }
        return;
    }
    const Words<W> s = ld_words<W>(own + rb), same = ld_words<W>(oth + rb);
    const Words<W> up = ld_words<W>(oth + (z * m.ly + yu) * m.hx + h0), dn = ld_words<W>(oth + (z * m.ly + yd) * m.hx + h0);
    Words<W> zp{}, zm{};
    if (DIM == 3) {
        zp = ld_words<W>(oth + (zu * m.ly + y) * m.hx + h0);
        zm = ld_words<W>(oth + (zd * m.ly + y) * m.hx + h0);
    }
    const uint32_t ex = (uint8_t)oth[hrow + ho];
    Words<W> out = s;
    uint32_t changed = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const uint32_t sh = shifted_word<W>(same, i, ex, xp);
        uint32_t pat = sign_bits(xp ? sh : same.w[i], 0) | sign_bits(xp ? same.w[i] : sh, 1) |
                       sign_bits(up.w[i], 2) | sign_bits(dn.w[i], 3) | sign_bits(s.w[i], ND);
        if (DIM == 3) pat |= sign_bits(zp.w[i], 4) | sign_bits(zm.w[i], 5);
        uint32_t flip = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const nmmc_u4 r = sweep_draw<true>(m, box + 2 * (4 * i + k), sw, (uint32_t)chain);
            // proposal +1 when r.x's top bit is set: it differs from the spin when that bit equals
            // the spin's sign bit
            const bool differs = (int32_t)(r.x ^ (s.w[i] << (24 - 8 * k))) >= 0;
            if (differs && (r.y >> 9) < st[(pat >> (8 * k)) & 0xFFu]) flip |= 0xFEu << (8 * k);
        }
        out.w[i] = s.w[i] ^ flip;   // 0x01 <-> 0xFF
        changed |= flip;
    }
    if (changed) {
        if (W == 4)
            *reinterpret_cast<uint4*>(own + rb) = make_uint4(out.w[0], out.w[W > 1 ? 1 : 0], out.w[W > 2 ? 2 : 0], out.w[W > 3 ? 3 : 0]);
        else
            *reinterpret_cast<uint32_t*>(own + rb) = out.w[0];
    }
}

// Observables of the words: per direction the number of sites whose neighbour agrees minus those
// whose neighbour does not, and the sums of the spins, as integers (exact); one block covers the
// rows of k_measure's blocks and writes its partials in that layout, the energy with FP64 J.
template <int DIM, bool PERIODIC>
__global__ void __launch_bounds__(256)
k_measure_ising(const DevModel m, const int8_t* __restrict__ spins, const int* __restrict__ chains, int rows,
                int nblk_slice, double* __restrict__ partial) {
    constexpr int ND = 2 * DIM;
    const int ci = blockIdx.y, chain = chains[ci], b = blockIdx.x;
    const int z = b / nblk_slice, y0 = (b - z * nblk_slice) * rows, y1 = min(y0 + rows, m.ly);
    const size_t P = (size_t)m.nhalf_pad;
    const int wpr = m.hx >> 2, nw = 2 * (y1 - y0) * wpr;
    const int e4 = m.edge - m.edge % 4;
    int acc[ND + 3];   // agreement per direction; M, M of colour 0, sub4
#pragma unroll
    for (int k = 0; k < ND + 3; ++k) acc[k] = 0;
    for (int it = threadIdx.x; it < nw; it += blockDim.x) {
        const int colour = it & 1, rq = it >> 1;
        const int yy = rq / wpr, h0 = (rq - yy * wpr) * 4, y = y0 + yy, xp = (y + z + colour) & 1;
        const int8_t* own = spins + ((size_t)chain * 2 + colour) * P;
        const int8_t* oth = spins + ((size_t)chain * 2 + (colour ^ 1)) * P;
        const int hrow = (z * m.ly + y) * m.hx;
        const uint32_t s = __ldg(reinterpret_cast<const uint32_t*>(own + hrow + h0));
        const Words<1> same = ld_words<1>(oth + hrow + h0);
        int ho = xp ? h0 + 4 : h0 - 1, yu = y + 1, yd = y - 1, zu = z + 1, zd = z - 1;
        uint32_t keep = 0x80808080u;   // sites whose x-neighbour outside the word exists
        bool okU = true, okD = true, okF = true, okB = true;
        if (PERIODIC) {
            ho = ho < 0 ? m.hx - 1 : (ho >= m.hx ? 0 : ho);
            yu = yu == m.ly ? 0 : yu;
            yd = yd < 0 ? m.ly - 1 : yd;
            zu = zu == m.lz ? 0 : zu;
            zd = zd < 0 ? m.lz - 1 : zd;
        } else {
            if (ho < 0 || ho >= m.hx) {
                keep = xp ? 0x00808080u : 0x80808000u;
                ho = h0;
            }
            okU = yu < m.ly;
            okD = yd >= 0;
            okF = zu < m.lz;
            okB = zd >= 0;
        }
        const uint32_t sh = shifted_word<1>(same, 0, (uint8_t)__ldg(oth + hrow + ho), xp);
        auto agree = [&](uint32_t w, uint32_t mask) { return __popc(mask) - 2 * __popc((s ^ w) & mask); };
        const int a_sh = agree(sh, keep), a_same = agree(same.w[0], 0x80808080u);
        acc[0] += xp ? a_sh : a_same;
        acc[1] += xp ? a_same : a_sh;
        auto row_of = [&](int zz, int yr) { return __ldg(reinterpret_cast<const uint32_t*>(oth + (zz * m.ly + yr) * m.hx + h0)); };
        if (okU) acc[2] += agree(row_of(z, yu), 0x80808080u);
        if (okD) acc[3] += agree(row_of(z, yd), 0x80808080u);
        if (DIM == 3) {
            if (okF) acc[ND - 2] += agree(row_of(zu, y), 0x80808080u);
            if (okB) acc[ND - 1] += agree(row_of(zd, y), 0x80808080u);
        }
        const int sum = 4 - 2 * __popc(s & 0x80808080u);
        acc[ND] += sum;
        if (colour == 0) acc[ND + 1] += sum;
        const int z4 = DIM == 3 ? (z & 3) : 0;
        if ((z4 & 1) == 0) {   // sub4M (Old/lib/thermodynamics.cpp:138-163), C truncating remainders
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = 2 * (h0 + k) + xp;
                if (((x + y) & 3) == z4 && (y - x + e4) % 4 == z4) acc[ND + 2] += (s >> (8 * k + 7)) & 1 ? -1 : 1;
            }
        }
    }
    __shared__ int red[ND + 3][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < ND + 3; ++k) {
        const int v = __reduce_add_sync(0xffffffffu, acc[k]);
        if (lane == 0) red[k][warp] = v;
    }
    __syncthreads();
    double* out = partial + ((size_t)ci * gridDim.x + b) * kNP;
    if (threadIdx.x < kNP) {
        auto total = [&](int k) {
            int v = 0;
            for (int w = 0; w < 8; ++w) v += red[k][w];
            return v;
        };
        double v = 0.0;   // 0 e, 1 M, 4 subM, 7 sub4M; the other components and the charge are 0
        if (threadIdx.x == 0)
            for (int k = 0; k < ND; ++k) v += m.Jd[k] * total(k);
        if (threadIdx.x == 1) v = total(ND);
        if (threadIdx.x == 4) v = total(ND + 1);
        if (threadIdx.x == 7) v = total(ND + 2);
        out[threadIdx.x] = v;
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
// Unmasked checkerboard lattices whose rows hold whole words of a colour, every site +1 or -1.
bool ising_words_ok(const Ctx& c) { return c.ising && !c.masked && !c.m.general && c.m.hx % 4 == 0 && c.ising_empties == 0; }

size_t ising_table_bytes(const Ctx& c) { return ising_words_ok(c) ? (size_t)c.nchains * kItabMax * sizeof(uint32_t) : 0; }

int launch_ising_table(Ctx& c) {
    if (!c.d_itab) return NMMC_OK;
    // a capture records the launch in any case: its graph may be replayed after other points were
    // uploaded, and has not run yet
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    NMMC_CUDA(cudaStreamIsCapturing(c.stream, &cs));
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (!c.itab_stale && !capturing) return NMMC_OK;
    k_ising_table<<<c.nchains, kItabMax, 0, c.stream>>>(c.m, c.d_bh, c.d_itab);
    if (int rc = cuda_check(cudaGetLastError(), "k_ising_table")) return rc;
    if (!capturing) c.itab_stale = false;
    return NMMC_OK;
}

template <int DIM, bool PERIODIC, int W>
static void ising_words_launch_w(Ctx& c, const int* d_chains, int n, int colour, unsigned off) {
    const int items = c.m.hx / (4 * W) * c.m.ly * c.m.lz;
    launch_seq(c, k_ising_words<DIM, PERIODIC, W>, dim3((items + 255) / 256, n), 256, 0,
        c.m, (int8_t*)c.d_spins, c.d_bh, c.d_sweep, d_chains, c.d_itab, colour, off);
}

// 16 sites per thread (16-byte loads, 71 instructions per update against 105) where rows hold them
// and the launch still gives every SM 1024 threads; 4 otherwise. 24 chains of 64^3: 13.9 us a
// colour with 16, 15.8 us with 4.
template <int DIM, bool PERIODIC>
static void ising_words_launch_p(Ctx& c, const int* d_chains, int n, int colour, unsigned off) {
    const long threads16 = (long)c.m.nhalf / 16 * n;
    if (c.m.hx % 16 == 0 && threads16 >= 1024L * c.sm_count) ising_words_launch_w<DIM, PERIODIC, 4>(c, d_chains, n, colour, off);
    else ising_words_launch_w<DIM, PERIODIC, 1>(c, d_chains, n, colour, off);
}

void launch_ising_words(Ctx& c, const int* d_chains, int n, int colour, unsigned off) {
    if (c.dim == 3) c.periodic ? ising_words_launch_p<3, true>(c, d_chains, n, colour, off)
                               : ising_words_launch_p<3, false>(c, d_chains, n, colour, off);
    else c.periodic ? ising_words_launch_p<2, true>(c, d_chains, n, colour, off)
                    : ising_words_launch_p<2, false>(c, d_chains, n, colour, off);
}

void launch_measure_ising(Ctx& c, dim3 grid, const int* d_chains, int rows, int nblk_slice, double* partial) {
    const int8_t* sp = (const int8_t*)c.d_spins;
    if (c.dim == 3) {
        if (c.periodic) k_measure_ising<3, true><<<grid, 256, 0, c.stream>>>(c.m, sp, d_chains, rows, nblk_slice, partial);
        else k_measure_ising<3, false><<<grid, 256, 0, c.stream>>>(c.m, sp, d_chains, rows, nblk_slice, partial);
    } else {
        if (c.periodic) k_measure_ising<2, true><<<grid, 256, 0, c.stream>>>(c.m, sp, d_chains, rows, nblk_slice, partial);
        else k_measure_ising<2, false><<<grid, 256, 0, c.stream>>>(c.m, sp, d_chains, rows, nblk_slice, partial);
    }
}

}  // namespace nmmc
