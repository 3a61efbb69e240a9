// General interaction tables: any list of offsets with J and D per record, read as the
// reference reads them (Old/lib/field_type.cpp:49-71) and summed in file order like its
// neighbour lists (field_type.cpp:104-141, thermodynamics.cpp:17-69). Tables beyond the
// 2*dim axis neighbours (next-nearest, third-nearest, long-range exchange) cannot use the
// two-colour checkerboard, so the lattice is split into colour classes in which no two sites
// interact through any record (find_colouring, nmmc_host.cpp); one launch updates one class
// of every listed chain, gathering each site's neighbours record by record.
//
// The Philox draw of a site is the one the checkerboard kernels use (box index, sweep
// counter, chain), so only the order of the classes differs from them.
//
// Unmasked Heisenberg lattices are swept in class planes: per chain and class its sites in row
// order, one float4 (x, y, z, 0) each, gathered from the box layout by each call and written back.
// The neighbours of a class through one record are all of one other class, so a warp's gather
// through a record is one contiguous 16-byte load per lane; in the box layout it was three
// scalar loads at a stride of half the period with its own wrap and plane arithmetic. A class of
// 20 chains of 64^3, 18 records: 1360 -> 773 instructions per update, 34.6 -> 23.6 us (issue 61 %
// busy, DRAM 44 %: every launch reads the whole lattices, 84 MB). Tables of more than 36 records
// and other lattices keep the box layout (k_colour_sweep).
#include <algorithm>

#include "nmmc_kernels.cuh"

namespace nmmc {

// Site handled by thread t of colour class `colour`; false when the thread has none.
template <int DIM>
__device__ __forceinline__ bool colour_site(const DevModel& m, int colour, int t, int& x, int& y, int& z) {
    if (m.col_kind == 1) {   // x + b*y + c*z = colour (mod q): x steps by q along each row
        const int q = m.col_q;
        const int kx = (m.edge + q - 1) / q;
        const int row = t / kx, k = t - row * kx;
        if (row >= m.ly * m.lz) return false;
        z = (DIM == 3) ? row / m.ly : 0;
        y = row - z * m.ly;
        int r = (colour - m.col_b * y - m.col_c * z) % q;
        if (r < 0) r += q;
        x = r + k * q;
    } else {                 // (x, y, z) = (cx, cy, cz) (mod p)
        const int p = m.col_p;
        const int cx = colour % p, cy = (colour / p) % p, cz = (DIM == 3) ? colour / (p * p) : 0;
        const int kx = (m.edge - cx + p - 1) / p, ky = (m.ly - cy + p - 1) / p;
        const int kz = (DIM == 3) ? (m.lz - cz + p - 1) / p : 1;
        const int k = t % kx, rest = t / kx;
        const int jy = rest % ky, jz = rest / ky;
        if (jz >= kz) return false;
        x = cx + k * p;
        y = cy + jy * p;
        z = cz + jz * p;
    }
    return x < m.edge;
}

// Neighbour of (x, y, z) through record offset o: its box coordinates, or false when it falls
// off an open boundary or is the site itself (the reference skips i == j). On periodic
// lattices the offsets are stored wrapped into [0, edge) and o.w marks a record that wraps
// onto the site itself, so the wrap is one conditional subtraction per axis.
template <int DIM, bool PERIODIC>
__device__ __forceinline__ bool general_neighbour(const DevModel& m, int x, int y, int z, int4 o, int& qx,
                                                  int& qy, int& qz) {
    qx = x + o.x;
    qy = y + o.y;
    qz = (DIM == 3) ? z + o.z : 0;
    if (PERIODIC) {
        const int e = m.edge;
        qx -= (qx >= e) ? e : 0;
        qy -= (qy >= e) ? e : 0;
        if (DIM == 3) qz -= (qz >= e) ? e : 0;
    } else {
        if (qx < 0 || qx >= m.edge || qy < 0 || qy >= m.edge) return false;
        if (DIM == 3 && (qz < 0 || qz >= m.edge)) return false;
    }
    return o.w == 0;
}

__device__ __forceinline__ size_t plane_index(const DevModel& m, int x, int y, int z) {
    return (size_t)(z * m.ly + y) * m.hx + (x >> 1);
}

// Records per batch of the gathers: the neighbour loads of kRecBatch records are issued
// before any of their terms is added, so their latencies overlap; the terms are still added
// one record at a time in file order.
constexpr int kRecBatch = 4;

// Local field of the sweep, FP32, records in file order: H + sum_r J_r s_r + s_r x Ds_r.
// Sites outside a particle hold 0 and add nothing. Ising: hx only.
template <int DIM, bool PERIODIC, bool ISING>
__device__ __forceinline__ void general_field(const DevModel& m, const void* __restrict__ spins_v, int chain,
                                              int x, int y, int z, float4 p, float& hx, float& hy, float& hz) {
    const size_t P = (size_t)m.nhalf_pad;
    const int8_t* si = (const int8_t*)spins_v + (size_t)chain * 2 * P;
    const float* sf = (const float*)spins_v + (size_t)chain * 2 * 3 * P;
    hx = p.y;
    hy = p.z;
    hz = p.w;
    const int ngen = m.ngen;
    for (int r0 = 0; r0 < ngen; r0 += kRecBatch) {
        float vx[kRecBatch], vy[kRecBatch], vz[kRecBatch];
        bool ok[kRecBatch];
#pragma unroll
        for (int u = 0; u < kRecBatch; ++u) {
            const int r = r0 + u;
            int qx, qy, qz;
            ok[u] = r < ngen && general_neighbour<DIM, PERIODIC>(m, x, y, z, __ldg(&m.g_off[r]), qx, qy, qz);
            vx[u] = vy[u] = vz[u] = 0.0f;
            if (ok[u]) {
                const size_t c2 = (size_t)((qx + qy + qz) & 1);
                const size_t j = plane_index(m, qx, qy, qz);
                if (ISING) {
                    vx[u] = (float)si[c2 * P + j];
                } else {
                    const float* pl = sf + c2 * 3 * P;
                    vx[u] = pl[j];
                    vy[u] = pl[P + j];
                    vz[u] = pl[2 * P + j];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kRecBatch; ++u) {
            if (!ok[u]) continue;
            const float4 js = __ldg(&m.g_js[r0 + u]);
            const float sx = vx[u], sy = vy[u], sz = vz[u];
            hx = fmaf(js.x, sx, hx);
            if (!ISING) {
                hy = fmaf(js.x, sy, hy);
                hz = fmaf(js.x, sz, hz);
                hx = fmaf(sy, js.w, fmaf(-sz, js.z, hx));   // s x Ds
                hy = fmaf(sz, js.y, fmaf(-sx, js.w, hy));
                hz = fmaf(sx, js.z, fmaf(-sy, js.y, hz));
            }
        }
    }
}

// One colour class of every listed chain (grid.y = list position).
template <int DIM, bool PERIODIC, bool MASKED, bool ISING>
__global__ void __launch_bounds__(256)
k_colour_sweep(const DevModel m, void* spins_v, const uint8_t* __restrict__ mask,
               const float4* __restrict__ bh, const unsigned long long* sweep,
               const int* __restrict__ chains, int colour, unsigned off, bool early) {
    if (early) seq_next();
    seq_wait();
    const int chain = chains[blockIdx.y];
    int x, y, z;
    if (!colour_site<DIM>(m, colour, blockIdx.x * blockDim.x + threadIdx.x, x, y, z)) return;
    const int c2 = (x + y + z) & 1;
    const size_t P = (size_t)m.nhalf_pad;
    const size_t i = plane_index(m, x, y, z);
    if (MASKED && !mask[((size_t)chain * 2 + c2) * P + i]) return;
    const float4 p = bh[chain];
    const uint32_t box = (uint32_t)(x + m.edge * (y + m.edge * z));
    const nmmc_u4 r = sweep_draw(m, box, sweep[chain] + off, (uint32_t)chain);
    float hx, hy, hz;
    general_field<DIM, PERIODIC, ISING>(m, spins_v, chain, x, y, z, p, hx, hy, hz);
    if (!early) seq_next();
    if (ISING) {
        int8_t* own = (int8_t*)spins_v + ((size_t)chain * 2 + c2) * P + i;
        float t;
        if (ising_try(hx, (float)*own, p, r, t)) *own = (int8_t)t;
    } else {
        float* pl = (float*)spins_v + ((size_t)chain * 2 + c2) * 3 * P;
        float tx, ty, tz;
        if (heis_try(hx, hy, hz, pl[i], pl[P + i], pl[2 * P + i], p, r, tx, ty, tz)) {
            pl[i] = tx;
            pl[P + i] = ty;
            pl[2 * P + i] = tz;
        }
    }
}

// ------------------------------------------------------------------------------------------
// Class planes of unmasked Heisenberg lattices
// ------------------------------------------------------------------------------------------
// Cells of a class: kind 1 (x + b y + c z mod q) every row's x = r, r + q, ...; kind 2 (product)
// every axis' residue cx, cx + p, .... Each class has room for the longest; cells whose site
// would lie outside the box are never used. Divisions are by multiplication: n / d =
// __umulhi(n, ceil(2^32 / d)) for n * d < 2^32 and d > 1.
struct Div32 { uint32_t mul; int d; };
struct ClassShape {
    int kx, ky, kz, cells;
    int step;                // q (kind 1) or p (kind 2)
    Div32 by_step, by_kx, by_ky;
    size_t chain;            // float4 of a chain: every class, and one zero cell past them
};

__device__ __forceinline__ unsigned div32(unsigned n, const Div32& d) { return d.mul ? __umulhi(n, d.mul) : n; }

static Div32 make_div(int d) { return Div32{d <= 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d), d}; }

static ClassShape class_shape(const Ctx& c) {
    ClassShape s;
    s.step = c.m.col_kind == 1 ? c.m.col_q : c.m.col_p;
    s.kx = (c.edge + s.step - 1) / s.step;
    s.ky = c.m.col_kind == 1 ? c.m.ly : s.kx;
    s.kz = c.dim == 2 ? 1 : (c.m.col_kind == 1 ? c.m.lz : s.kx);
    s.cells = s.kx * s.ky * s.kz;
    s.by_step = make_div(s.step);
    s.by_kx = make_div(s.kx);
    s.by_ky = make_div(s.ky);
    s.chain = (size_t)s.cells * c.m.col_q + 1;
    return s;
}

// Site of cell t of class `cls`; false where the cell has none.
template <int DIM>
__device__ __forceinline__ bool class_site(const DevModel& m, const ClassShape& s, int cls, int t, int& x, int& y,
                                           int& z) {
    const int row = div32(t, s.by_kx), k = t - row * s.kx;
    const int jz = DIM == 3 ? div32(row, s.by_ky) : 0, jy = row - jz * s.ky;
    if (m.col_kind == 1) {
        y = jy;
        z = jz;
        const int q = m.col_q;   // x = cls - b y - c z (mod q)
        const unsigned w = (unsigned)(m.col_b * y + m.col_c * z);
        int r = cls - (int)(w - div32(w, s.by_step) * q);
        r += r < 0 ? q : 0;
        x = r + k * q;
    } else {
        const int p = m.col_p;
        x = cls % p + k * p;
        y = (cls / p) % p + jy * p;
        z = DIM == 3 ? cls / (p * p) + jz * p : 0;
    }
    return jz < s.kz && x < m.edge && y < m.ly && z < m.lz;
}

// A table in the form the class kernels take, as a kernel parameter: a neighbour's index in the
// chain's class planes is base (its class, the same for every site of a class) + the term of its
// row (one of `na` distinct (oy, oz)) + the term of its column (one of `nb` distinct ox). A thread
// computes its site's na + nb terms once and keeps them in its own column of shared memory.
constexpr int kClassBatch = 9, kClassRecs = 4 * kClassBatch, kClassRows = 16, kClassCols = 8;
struct ClassTable {
    int n, na, nb;                 // n: records, padded to whole batches with records of J = D = 0
    int2 row[kClassRows];          // distinct (oy, oz), wrapped into [0, edge) on periodic lattices
    int col[kClassCols];           // distinct ox
    int2 at[kClassRecs];           // per record: its row and its column term (offsets into the slots)
    float4 j[kClassRecs];          // J, D
};
struct ClassBase { int b[kClassRecs]; };   // per record: first cell of the neighbours' class
constexpr int kNoCell = -(1 << 30);        // a term that makes the index negative: past an open edge

// The site's terms into its column of `slots` ([slot][256]; the last slot holds 0, for padding).
template <int DIM, bool PERIODIC>
__device__ __forceinline__ void class_terms(const DevModel& m, const ClassShape& s, const ClassTable& t, int x, int y,
                                            int z, int* slots) {
    const unsigned e = m.edge;
    const bool lin = m.col_kind == 1;
#pragma unroll 3
    for (int i = 0; i < t.na; ++i) {
        unsigned qy = y + t.row[i].x, qz = DIM == 3 ? z + t.row[i].y : 0;
        bool ok = true;
        if (PERIODIC) {   // offsets are in [0, edge): one subtraction wraps, and underflows where it must not
            qy = min(qy, qy - e);
            if (DIM == 3) qz = min(qz, qz - e);
        } else {
            ok = qy < e && (DIM == 2 || qz < e);
        }
        if (!lin) {
            qy = div32(qy, s.by_step);
            if (DIM == 3) qz = div32(qz, s.by_step);
        }
        slots[i * 256] = ok ? (int)((qz * s.ky + qy) * s.kx) : kNoCell;
    }
#pragma unroll 3
    for (int i = 0; i < t.nb; ++i) {
        unsigned qx = x + t.col[i];
        if (PERIODIC) qx = min(qx, qx - e);
        slots[(t.na + i) * 256] = PERIODIC || qx < e ? (int)div32(qx, s.by_step) : kNoCell;
    }
    slots[(t.na + t.nb) * 256] = 0;
}

// Adds the records' terms to the field in file order, the loads of a batch before its terms.
// SWEEP: s_j x Ds (the sweep's convention), else De x s_j (the energy's). Products of a zero J or D
// change nothing; neighbours past an open edge read the zero cell.
template <bool PERIODIC, bool SWEEP>
__device__ __forceinline__ void class_field(const ClassTable& t, const ClassBase& base, const float4* __restrict__ plane,
                                            int zero, const int* slots, float& hx, float& hy, float& hz) {
    constexpr int B = kClassBatch;
#pragma unroll
    for (int r0 = 0; r0 < kClassRecs; r0 += B) {
        if (r0 >= t.n) break;
        float4 v[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int2 at = t.at[r0 + u];
            int i = base.b[r0 + u] + slots[at.x] + slots[at.y];
            if (!PERIODIC) i = i < 0 ? zero : i;
            v[u] = plane[i];
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const float4 j = t.j[r0 + u];
            const float sx = v[u].x, sy = v[u].y, sz = v[u].z;
            hx = fmaf(j.x, sx, hx);
            hy = fmaf(j.x, sy, hy);
            hz = fmaf(j.x, sz, hz);
            if (SWEEP) {
                hx = fmaf(sy, j.w, fmaf(-sz, j.z, hx));
                hy = fmaf(sz, j.y, fmaf(-sx, j.w, hy));
                hz = fmaf(sx, j.z, fmaf(-sy, j.y, hz));
            } else {
                hx = fmaf(j.z, sz, fmaf(-j.w, sy, hx));
                hy = fmaf(j.w, sx, fmaf(-j.y, sz, hy));
                hz = fmaf(j.y, sy, fmaf(-j.z, sx, hz));
            }
        }
    }
}

// One colour class of every listed chain, in its class planes.
template <int DIM, bool PERIODIC>
__global__ void __launch_bounds__(256, 4)
k_class_sweep(const __grid_constant__ DevModel m, const ClassShape s, const __grid_constant__ ClassTable t,
              const __grid_constant__ ClassBase base, float4* planes, const float4* __restrict__ bh,
              const unsigned long long* sweep, const int* __restrict__ chains, int colour, unsigned off) {
    extern __shared__ int cl_slots[];
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    int x, y, z;
    const bool mine = cell < s.cells && class_site<DIM>(m, s, colour, cell, x, y, z);
    int* const slots = cl_slots + threadIdx.x;
    if (mine) class_terms<DIM, PERIODIC>(m, s, t, x, y, z, slots);   // before the wait: parameters only
    seq_begin();
    if (!mine) return;
    const int chain = chains[blockIdx.y];
    float4* const plane = planes + (size_t)chain * s.chain;
    float4* const own = plane + (size_t)colour * s.cells + cell;
    const float4 p = bh[chain];
    const uint32_t box = (uint32_t)(x + m.edge * (y + m.edge * z));
    const nmmc_u4 r = sweep_draw<true>(m, box, sweep[chain] + off, (uint32_t)chain);
    float hx = p.y, hy = p.z, hz = p.w;
    class_field<PERIODIC, true>(t, base, plane, (int)s.chain - 1, slots, hx, hy, hz);
    const float4 v = *own;
    float tx, ty, tz;
    if (heis_try(hx, hy, hz, v.x, v.y, v.z, p, r, tx, ty, tz)) *own = make_float4(tx, ty, tz, 0.0f);
}

// Between the box layout and the class planes of the listed chains.
template <int DIM>
__global__ void __launch_bounds__(256)
k_class_copy(const DevModel m, const ClassShape s, float4* planes, float* spins,
             const int* __restrict__ chains, int to_class) {
    seq_begin();
    const int chain = chains[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.col_q * s.cells) return;
    const int cls = i / s.cells;
    int x, y, z;
    if (!class_site<DIM>(m, s, cls, i - cls * s.cells, x, y, z)) return;
    const size_t P = (size_t)m.nhalf_pad;
    float* b = spins + ((size_t)chain * 2 + ((x + y + z) & 1)) * 3 * P + plane_index(m, x, y, z);
    float4* q = planes + (size_t)chain * s.chain + i;
    if (to_class) {
        *q = make_float4(b[0], b[P], b[2 * P], 0.0f);
    } else {
        const float4 v = *q;
        b[0] = v.x;
        b[P] = v.y;
        b[2 * P] = v.z;
    }
}

// The table's energy term over the class planes: block b of a chain takes an equal run of class
// `cls`'s cells and adds its sum to slot 0 of the measurement's block b (as k_energy_general; FP32
// terms, FP64 across warps). One launch per class: the launches of a stream follow one another.
template <int DIM, bool PERIODIC>
__global__ void __launch_bounds__(256, 4)
k_class_energy(const __grid_constant__ DevModel m, const ClassShape s, const __grid_constant__ ClassTable t,
               const __grid_constant__ ClassBase base, const float4* planes, const int* __restrict__ chains,
               int cls, int nblk, float scale, double* partial) {
    seq_begin();
    extern __shared__ int cl_slots[];
    __shared__ float red[8];
    const int chain = chains[blockIdx.y];
    const float4* const plane = planes + (size_t)chain * s.chain;
    int* const slots = cl_slots + threadIdx.x;
    float acc = 0.0f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.cells; i += gridDim.x * blockDim.x) {
        int x, y, z;
        if (!class_site<DIM>(m, s, cls, i, x, y, z)) continue;
        class_terms<DIM, PERIODIC>(m, s, t, x, y, z, slots);
        const float4 v = plane[(size_t)cls * s.cells + i];
        float fx = 0.0f, fy = 0.0f, fz = 0.0f;
        class_field<PERIODIC, false>(t, base, plane, (int)s.chain - 1, slots, fx, fy, fz);
        acc += fmaf(v.x, fx, fmaf(v.y, fy, v.z * fz));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += (double)red[w];
        partial[((size_t)blockIdx.y * nblk + blockIdx.x) * kNP] += scale * tot;
    }
}

// The records a class kernel takes, in file order: all but those that land on the site itself. The
// energy of a table of +-o pairs (J(o) = J(-o), D(o) = -D(-o)) counts every bond from both ends with
// the same value, so the first record of each pair stands for both (class_energy_scale 2).
static bool class_paired(const Ctx& c, size_t r, size_t q) {
    const int4 a = c.h_goff[r], b = c.h_goff[q];
    const int e = c.edge;
    auto opposite = [&](int u, int v) { return c.periodic ? (u + v) % e == 0 : u + v == 0; };
    const float4 ja = c.h_gje[r], jb = c.h_gje[q];
    return opposite(a.x, b.x) && opposite(a.y, b.y) && opposite(a.z, b.z) && ja.x == jb.x && ja.y == -jb.y &&
           ja.z == -jb.z && ja.w == -jb.w;
}

static bool class_halves(const Ctx& c, std::vector<size_t>& first) {
    const size_t n = c.h_goff.size();
    std::vector<char> used(n, 0);
    first.clear();
    for (size_t r = 0; r < n; ++r) {
        if (used[r] || c.h_goff[r].w) continue;
        size_t q = r + 1;
        while (q < n && (used[q] || !class_paired(c, r, q))) ++q;
        if (q == n) return false;
        used[q] = 1;
        first.push_back(r);
    }
    return true;
}

static std::vector<size_t> class_records(const Ctx& c, bool sweep) {
    std::vector<size_t> recs;
    if (!sweep && c.h_goff.size() <= 2 * kClassRecs && class_halves(c, recs)) return recs;
    recs.clear();
    for (size_t r = 0; r < c.h_goff.size(); ++r)
        if (!c.h_goff[r].w) recs.push_back(r);
    return recs;
}

static float class_energy_scale(const Ctx& c) {
    std::vector<size_t> recs;
    return c.h_goff.size() <= 2 * kClassRecs && class_halves(c, recs) ? 2.0f : 1.0f;
}

// The class form of the context's records (js: in the wanted DMI convention); false where it has
// more records, rows or columns than the kernels take.
static bool class_table(const Ctx& c, bool sweep, ClassTable& t) {
    t.n = 0;
    t.na = t.nb = 0;
    for (size_t r : class_records(c, sweep)) {
        const int4 o = c.h_goff[r];
        if (t.n == kClassRecs) return false;
        int a = 0, b = 0;
        while (a < t.na && (t.row[a].x != o.y || t.row[a].y != o.z)) ++a;
        if (a == t.na) {
            if (t.na == kClassRows) return false;
            t.row[t.na++] = make_int2(o.y, o.z);
        }
        while (b < t.nb && t.col[b] != o.x) ++b;
        if (b == t.nb) {
            if (t.nb == kClassCols) return false;
            t.col[t.nb++] = o.x;
        }
        const float4 e = c.h_gje[r];
        t.j[t.n] = sweep && c.dmi_sign ? make_float4(e.x, -e.y, -e.z, -e.w) : e;
        t.at[t.n++] = make_int2(a, b);
    }
    for (int r = 0; r < t.n; ++r) t.at[r] = make_int2(t.at[r].x * 256, (t.na + t.at[r].y) * 256);
    while (t.n % kClassBatch) {   // padding: the zero cell, by the zero slot
        t.at[t.n] = make_int2((t.na + t.nb) * 256, (t.na + t.nb) * 256);
        t.j[t.n++] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    return true;
}

static ClassBase class_base(const Ctx& c, const ClassShape& s, bool sweep, int cls) {
    ClassBase base{};
    const int q = c.m.col_q, p = c.m.col_p;
    int n = 0;
    for (size_t r : class_records(c, sweep)) {
        const int4 o = c.h_goff[r];
        int k;
        if (c.m.col_kind == 1) {
            k = (int)(((cls + o.x + (long)c.m.col_b * o.y + (long)c.m.col_c * o.z) % q + q) % q);
        } else {
            auto mod = [&](int v) { return (v % p + p) % p; };
            k = mod(cls % p + o.x) + p * mod((cls / p) % p + o.y) + (c.dim == 3 ? p * p * mod(cls / (p * p) + o.z) : 0);
        }
        base.b[n++] = k * s.cells;
    }
    while (n < kClassRecs) base.b[n++] = (int)s.chain - 1;
    return base;
}

static bool use_class(const Ctx& c) {
    if (!c.m.general || c.masked || c.ising || c.class_no_memory || c.half_kernel == 1) return false;
    const ClassShape s = class_shape(c);
    ClassTable t;
    // indices below the no-cell marker; the division by multiplication
    return (long long)s.cells * c.m.col_q < (1LL << 29) && (long long)s.cells * s.kx < (1LL << 32) &&
           (long long)(s.ky * s.kz) * s.ky < (1LL << 32) && (long long)(c.m.col_q + 1) * 2 * c.edge * s.step < (1LL << 32) &&
           class_table(c, true, t);
}

// The class planes, allocated at the first sweep; without the memory, and in a stream capture that
// comes before it, the sweeps stay in the box.
bool class_ready(Ctx& c) {
    if (!use_class(c)) return false;
    if (c.d_class) return true;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c.stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return false;
    const ClassShape s = class_shape(c);
    if (cudaMalloc(&c.d_class, (size_t)c.nchains * s.chain * sizeof(float4)) != cudaSuccess ||
        cudaMemsetAsync(c.d_class, 0, (size_t)c.nchains * s.chain * sizeof(float4), c.stream) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(c.d_class);
        c.d_class = nullptr;
        c.class_no_memory = true;
        return false;
    }
    return true;
}

static int class_copy(Ctx& c, const int* d_chains, int n, bool to_class) {
    const ClassShape s = class_shape(c);
    const dim3 grid((c.m.col_q * s.cells + 255) / 256, n);
    if (c.dim == 3) launch_seq(c, k_class_copy<3>, grid, 256, 0, c.m, s, c.d_class, (float*)c.d_spins, d_chains, to_class);
    else launch_seq(c, k_class_copy<2>, grid, 256, 0, c.m, s, c.d_class, (float*)c.d_spins, d_chains, to_class);
    return cuda_check(cudaGetLastError(), "k_class_copy");
}

static int class_sweeps(Ctx& c, const int* d_chains, int n, int nsweeps) {
    const ClassShape s = class_shape(c);
    if (int rc = class_copy(c, d_chains, n, true)) return rc;
    const dim3 grid((s.cells + 255) / 256, n);
    auto kern = c.dim == 3 ? (c.periodic ? k_class_sweep<3, true> : k_class_sweep<3, false>)
                           : (c.periodic ? k_class_sweep<2, true> : k_class_sweep<2, false>);
    ClassTable t;
    class_table(c, true, t);
    std::vector<ClassBase> base;
    for (int colour = 0; colour < c.m.col_q; ++colour) base.push_back(class_base(c, s, true, colour));
    const size_t smem = (size_t)(t.na + t.nb + 1) * 256 * sizeof(int);   // at most 25 KB
    for (int k = 0; k < nsweeps; ++k)
        for (int colour = 0; colour < c.m.col_q; ++colour)
            launch_seq(c, kern, grid, 256, smem, c.m, s, t, base[colour], c.d_class, c.d_bh, c.d_sweep, d_chains, colour,
                                                (unsigned)k);
    if (int rc = cuda_check(cudaGetLastError(), "k_class_sweep")) return rc;
    if (int rc = class_copy(c, d_chains, n, false)) return rc;
    c.planes_fresh = true;
    return launch_advance(c, d_chains, n, nsweeps);
}

// Threads per chain for one colour class (the largest class).
static int colour_threads(const Ctx& c) {
    const DevModel& m = c.m;
    if (m.col_kind == 1) return m.ly * m.lz * ((m.edge + m.col_q - 1) / m.col_q);
    const int k = (m.edge + m.col_p - 1) / m.col_p;
    return k * k * (c.dim == 3 ? k : 1);
}

template <int DIM, bool PERIODIC, bool MASKED, bool ISING>
static void colour_launch(Ctx& c, const int* d_chains, int n, int colour, unsigned off) {
    dim3 grid((colour_threads(c) + 255) / 256, n);
    // The next launch's blocks move in behind this one's from the start where those come in several
    // rounds; where all are resident at once, only after the gathers: while they wait they keep blocks of
    // this launch from being spread evenly over the SMs (173 Ising chains of 12^3, 5 sweeps: 313 us at the
    // start, 213 after the gathers, 268 by plain launches; 2314 of them 868, 903 and 976).
    const bool early = (long long)grid.x * n > 16LL * c.sm_count;
    launch_seq(c, k_colour_sweep<DIM, PERIODIC, MASKED, ISING>, grid, 256, 0,
        c.m, c.d_spins, c.d_mask, c.d_bh, c.d_sweep, d_chains, colour, off, early);
}

using ColourFn = void (*)(Ctx&, const int*, int, int, unsigned);

template <int DIM, bool PERIODIC>
static ColourFn pick_colour_pm(const Ctx& c) {
    if (c.ising) return c.masked ? colour_launch<DIM, PERIODIC, true, true> : colour_launch<DIM, PERIODIC, false, true>;
    return c.masked ? colour_launch<DIM, PERIODIC, true, false> : colour_launch<DIM, PERIODIC, false, false>;
}

int launch_colour_sweeps(Ctx& c, const int* d_chains, int n, int nsweeps) {
    // A class launch saves a quarter (4 classes in 2-D) to two fifths (6 in 3-D) of a box launch, and the
    // two copies cost as much as six of those quarters: 6944 chains of 24^2, one sweep, 157 us in class
    // planes and 134 in the box, two sweeps 237 and 246; 36 of 48^3 (6 classes) one sweep 172 and 222.
    if ((long long)nsweeps * c.m.col_q > 4 && class_ready(c)) return class_sweeps(c, d_chains, n, nsweeps);
    ColourFn f = (c.dim == 3) ? (c.periodic ? pick_colour_pm<3, true>(c) : pick_colour_pm<3, false>(c))
                              : (c.periodic ? pick_colour_pm<2, true>(c) : pick_colour_pm<2, false>(c));
    for (int s = 0; s < nsweeps; ++s)
        for (int colour = 0; colour < c.m.col_q; ++colour) f(c, d_chains, n, colour, (unsigned)s);
    int rc = cuda_check(cudaGetLastError(), "colour-sweep launch");
    if (rc) return rc;
    return launch_advance(c, d_chains, n, nsweeps);
}

// ------------------------------------------------------------------------------------------
// Energy term of a general table (thermodynamics.cpp:71-96): sum_i s_i . sum_r (J_r s_r +
// De_r x s_r), added to slot 0 of the partial sums the measurement kernel wrote for the same
// blocks (same rows-per-block split), so the finalisation is unchanged.
// ------------------------------------------------------------------------------------------
template <int DIM, bool PERIODIC, bool MASKED, bool ISING, typename RT>
__global__ void __launch_bounds__(256)
k_energy_general(const DevModel m, const void* __restrict__ spins_v, const uint8_t* __restrict__ mask,
                 const int* __restrict__ chains, int rows, int nblk_slice, int nblk_total,
                 double* __restrict__ partial) {
    const int ci = blockIdx.y;
    const int chain = chains[ci];
    const int b = blockIdx.x;
    const int z = b / nblk_slice;
    const int y0 = (b - z * nblk_slice) * rows;
    const int y1 = min(y0 + rows, m.ly);
    const int nsite = (y1 - y0) * m.edge;
    const size_t P = (size_t)m.nhalf_pad;
    auto load = [&](int x, int y, int zz, RT& s0, RT& s1, RT& s2) {
        const int c2 = (x + y + zz) & 1;
        const size_t i = plane_index(m, x, y, zz);
        if (ISING) {
            s0 = RT(((const int8_t*)spins_v)[((size_t)chain * 2 + c2) * P + i]);
            s1 = s2 = RT(0);
        } else {
            const float* pl = (const float*)spins_v + ((size_t)chain * 2 + c2) * 3 * P;
            s0 = RT(pl[i]);
            s1 = RT(pl[P + i]);
            s2 = RT(pl[2 * P + i]);
        }
    };
    RT acc = RT(0);
    for (int t = threadIdx.x; t < nsite; t += blockDim.x) {
        const int yy = t / m.edge, y = y0 + yy, x = t - yy * m.edge;
        if (MASKED && !mask[((size_t)chain * 2 + ((x + y + z) & 1)) * P + plane_index(m, x, y, z)]) continue;
        RT s0, s1, s2;
        load(x, y, z, s0, s1, s2);
        RT f0 = RT(0), f1 = RT(0), f2 = RT(0);
        const int ngen = m.ngen;
        for (int r0 = 0; r0 < ngen; r0 += kRecBatch) {
            RT a0[kRecBatch], a1[kRecBatch], a2[kRecBatch];
            bool ok[kRecBatch];
#pragma unroll
            for (int u = 0; u < kRecBatch; ++u) {   // loads of the batch first, terms in file order
                const int r = r0 + u;
                int qx, qy, qz;
                ok[u] = r < ngen && general_neighbour<DIM, PERIODIC>(m, x, y, z, __ldg(&m.g_off[r]), qx, qy, qz);
                a0[u] = a1[u] = a2[u] = RT(0);
                if (ok[u]) load(qx, qy, qz, a0[u], a1[u], a2[u]);
            }
#pragma unroll
            for (int u = 0; u < kRecBatch; ++u) {
                if (!ok[u]) continue;
                const int r = r0 + u;
                const RT n0 = a0[u], n1 = a1[u], n2 = a2[u];
                RT J, d0, d1, d2;
                if (sizeof(RT) == 8) {
                    J = RT(m.g_jed[4 * r]);
                    d0 = RT(m.g_jed[4 * r + 1]);
                    d1 = RT(m.g_jed[4 * r + 2]);
                    d2 = RT(m.g_jed[4 * r + 3]);
                } else {
                    const float4 je = __ldg(&m.g_je[r]);
                    J = RT(je.x);
                    d0 = RT(je.y);
                    d1 = RT(je.z);
                    d2 = RT(je.w);
                }
                f0 += J * n0;
                if (!ISING) {
                    f1 += J * n1;
                    f2 += J * n2;
                    f0 += d1 * n2 - d2 * n1;   // De x s_j
                    f1 += d2 * n0 - d0 * n2;
                    f2 += d0 * n1 - d1 * n0;
                }
            }
        }
        acc += s0 * f0 + s1 * f1 + s2 * f2;
    }
    // warp sums in the mode's type (FP32 mode: as the measurement kernels), FP64 across warps
    __shared__ RT red[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RT v = acc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += (double)red[w];
        partial[((size_t)ci * nblk_total + b) * kNP] += tot;
    }
}

template <int DIM, bool PERIODIC, bool MASKED, bool ISING>
static void energy_launch(Ctx& c, const int* d_chains, int n, int rows, int nblk_slice, int nblk_total,
                          double* partial) {
    dim3 grid(nblk_slice * c.m.lz, n);
    if (c.measure_fp64)
        k_energy_general<DIM, PERIODIC, MASKED, ISING, double><<<grid, 256, 0, c.stream>>>(
            c.m, c.d_spins, c.d_mask, d_chains, rows, nblk_slice, nblk_total, partial);
    else
        k_energy_general<DIM, PERIODIC, MASKED, ISING, float><<<grid, 256, 0, c.stream>>>(
            c.m, c.d_spins, c.d_mask, d_chains, rows, nblk_slice, nblk_total, partial);
}

template <int DIM, bool PERIODIC>
static void energy_pm(Ctx& c, const int* d, int n, int rows, int nbs, int nbt, double* partial) {
    if (c.ising) {
        if (c.masked) energy_launch<DIM, PERIODIC, true, true>(c, d, n, rows, nbs, nbt, partial);
        else energy_launch<DIM, PERIODIC, false, true>(c, d, n, rows, nbs, nbt, partial);
    } else {
        if (c.masked) energy_launch<DIM, PERIODIC, true, false>(c, d, n, rows, nbs, nbt, partial);
        else energy_launch<DIM, PERIODIC, false, false>(c, d, n, rows, nbs, nbt, partial);
    }
}

int launch_energy_general(Ctx& c, const int* d_chains, int n, int rows, int nblk_slice, int nblk_total,
                          double* partial) {
    // In class planes for 3-D tables and a million sites on (36 chains of 48^3: 177 us with the gather,
    // 240 in the box); below, a launch per class costs more than it saves (21 of 24^3: 57 and 50 us), and in
    // 2-D few records share a row (6944 of 24^2: 345 and 267 us, 1736 of 48^2 177 and 158).
    // Not for a caller's own scratch (nmmc_measure_static): its launches may be replayed from a graph
    // while the context sweeps in those planes.
    if (!c.measure_fp64 && c.dim == 3 && (long long)n * c.box_sites >= 1000000 && partial == c.d_partial && use_class(c) && c.d_class) {
        // a sample step's sweeps have left the listed chains' class planes current
        if (!c.planes_fresh)
            if (int rc = class_copy(c, d_chains, n, true)) return rc;
        auto kern = c.periodic ? k_class_energy<3, true> : k_class_energy<3, false>;
        const ClassShape s = class_shape(c);
        ClassTable t;
        class_table(c, false, t);
        const size_t smem = (size_t)(t.na + t.nb + 1) * 256 * sizeof(int);
        const int blocks = std::min(nblk_total, (s.cells + 255) / 256);
        for (int cls = 0; cls < c.m.col_q; ++cls)
            launch_seq(c, kern, dim3(blocks, n), 256, smem, c.m, s, t, class_base(c, s, false, cls), c.d_class, d_chains, cls,
                                                          nblk_total, class_energy_scale(c), partial);
        return cuda_check(cudaGetLastError(), "k_class_energy");
    }
    if (c.dim == 3) {
        if (c.periodic) energy_pm<3, true>(c, d_chains, n, rows, nblk_slice, nblk_total, partial);
        else energy_pm<3, false>(c, d_chains, n, rows, nblk_slice, nblk_total, partial);
    } else {
        if (c.periodic) energy_pm<2, true>(c, d_chains, n, rows, nblk_slice, nblk_total, partial);
        else energy_pm<2, false>(c, d_chains, n, rows, nblk_slice, nblk_total, partial);
    }
    return cuda_check(cudaGetLastError(), "k_energy_general");
}

// ------------------------------------------------------------------------------------------
// dE probe with the general sweep's FP32 field.
// ------------------------------------------------------------------------------------------
template <int DIM, bool PERIODIC, bool ISING>
__global__ void k_delta_e_general(const DevModel m, const void* __restrict__ spins_v,
                                  const float4* __restrict__ bh, int chain, const int32_t* __restrict__ sites,
                                  const float* __restrict__ trial, int n, double* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int box = sites[t];
    const int x = box % m.edge, y = (box / m.edge) % m.edge, z = (DIM == 3) ? box / (m.edge * m.edge) : 0;
    const int c2 = (x + y + z) & 1;
    const size_t P = (size_t)m.nhalf_pad, i = plane_index(m, x, y, z);
    float hx, hy, hz;
    general_field<DIM, PERIODIC, ISING>(m, spins_v, chain, x, y, z, bh[chain], hx, hy, hz);
    if (ISING) {
        const float so = (float)((const int8_t*)spins_v)[((size_t)chain * 2 + c2) * P + i];
        out[t] = (double)(hx * (so - trial[3 * t]));
    } else {
        const float* pl = (const float*)spins_v + ((size_t)chain * 2 + c2) * 3 * P;
        out[t] = (double)heis_dE(hx, hy, hz, pl[i], pl[P + i], pl[2 * P + i], trial[3 * t], trial[3 * t + 1],
                                 trial[3 * t + 2]);
    }
}

int launch_delta_e_general(Ctx& c, int chain, const int32_t* d_sites, const float* d_trial, int n, double* d_out) {
    const int g = (n + 127) / 128;
#define NMMC_DEG(D, PR, IS) \
    k_delta_e_general<D, PR, IS><<<g, 128, 0, c.stream>>>(c.m, c.d_spins, c.d_bh, chain, d_sites, d_trial, n, d_out)
    if (c.dim == 3) {
        if (c.periodic) { if (c.ising) NMMC_DEG(3, true, true); else NMMC_DEG(3, true, false); }
        else { if (c.ising) NMMC_DEG(3, false, true); else NMMC_DEG(3, false, false); }
    } else {
        if (c.periodic) { if (c.ising) NMMC_DEG(2, true, true); else NMMC_DEG(2, true, false); }
        else { if (c.ising) NMMC_DEG(2, false, true); else NMMC_DEG(2, false, false); }
    }
#undef NMMC_DEG
    return cuda_check(cudaGetLastError(), "k_delta_e_general");
}

// ------------------------------------------------------------------------------------------
// Device records
// ------------------------------------------------------------------------------------------
int upload_general(Ctx& c) {
    const size_t n = c.h_gje.size();
    if (!n) return NMMC_OK;
    std::vector<float4> js(n);
    for (size_t r = 0; r < n; ++r) {   // sweep convention: s_j x D (reference) or D x s_j
        const float4& e = c.h_gje[r];
        js[r] = c.dmi_sign ? make_float4(e.x, -e.y, -e.z, -e.w) : e;
    }
    NMMC_CUDA(cudaMemcpyAsync(c.d_gjs, js.data(), n * sizeof(float4), cudaMemcpyHostToDevice, c.stream));
    return cuda_check(cudaStreamSynchronize(c.stream), "upload_general");
}

}  // namespace nmmc
