// fn_column.cuh -- noise evaluated along a column of a uniform grid.
//
// The specialised column kernels (fn_jit.cpp) give every lane one position across the
// grid's last axis and walk it along that axis, so all lanes of a warp share the last
// coordinate.  Where a node's position is still separable (its last component depends on the
// last grid axis alone, the others on the other axes alone), everything the lattice
// contributes changes only when that coordinate enters another cell, and everything that
// depends on the other axes never changes.  The structs below keep those parts in registers
// between steps.  What depends on the column's coordinate alone (cell, offset, easing curve)
// is the same for all lanes: the lanes compute 32 steps' worth at a time into shared memory,
// one step each, and every step reads its entry with one broadcast load.  A step then runs
// the reference's remaining arithmetic, the same operations in the same order on the same
// operands, so results equal the point functions of fn_device.cuh.
//
// Bound by: instruction issue.  A Perlin octave in 3D costs ~17 instructions a step (a packed
// fma per corner pair, packed lerps) against ~200 for the point function, whose integer
// hashing and gradient selection (the half-rate ALU pipe) move to the plane rebuild, ~115
// instructions once per cell.
#pragma once

#include "fn_device.cuh"

namespace fnd {

// Keeps a value the same but hides where it came from: computations on the result are not
// hoisted out of the (rare) branch they are needed in, where they would hold registers.
FND float opaque(float v)
{
    asm volatile("" : "+f"(v));
    return v;
}

FND float nan_() { return __int_as_float(0x7fffffff); }

// The gradient dot of one lattice corner as a function of the offset t along the last axis,
// for fixed offsets across it: dot = fma(s, t, g) with s in {-1, 0, 1}.  s * t is exact, so
// the fma rounds once, as the reference's sum of two signed offsets does (3D, 4D).
FND void grad_col3(int h, float x, float y, float& s, float& g)
{
    // the second offset is y (h & 12 == 0), x (h & 13 == 12) or the column's own; a zero
    // second offset and the column's signed weight are exclusive
    const bool takes_y = (h & 12) == 0, takes_x = (h & 13) == 12;
    const float u = flip((h & 8) ? y : x, h << 31), sign = flip(1.0f, h << 30);
    s = takes_y ? 0.0f : (takes_x ? 0.0f : sign);
    g = fmaf(takes_y ? y : (takes_x ? x : 0.0f), sign, u);
}
FND void grad_col4(int h, float x, float y, float z, float& s, float& g)
{
    const bool any34 = (h & 24) != 0, b4 = (h & 16) != 0, both34 = (h & 24) == 24;
    const float ab = flip(any34 ? x : y, h << 31) + flip(b4 ? y : z, h << 30);
    s = both34 ? 0.0f : flip(1.0f, h << 29);
    g = both34 ? ab + flip(z, h << 29) : ab;
}

// Cell bookkeeping shared by the columns.  prepare() fills the lane's table entry (offset,
// offset - 1, easing, cell) for the coordinate Z of step `lane` and returns the ballot of
// steps that enter another cell than the step before (a NaN cell always does).  enter() says
// whether the kept upper plane becomes the lower one (1, the usual step to the next cell) or
// both planes are new (0).
struct ColCell {
    float cell;
    int icell;
    FND void init() { cell = nan_(); icell = 0; }
    template <typename Ease>
    FND unsigned prepare(float4* tab, unsigned lane, float Z, Ease&& ease)
    {
        const float zs = floorf(Z), z0 = Z - zs;
        tab[lane] = make_float4(z0, z0 - 1.0f, ease(z0), zs);
        const float before = __shfl_up_sync(0xffffffffu, zs, 1);
        return __ballot_sync(0xffffffffu, zs != (lane ? before : cell));
    }
    FND int enter(float zs, int& zi)
    {
        zi = cvti(zs);
        const int from = (cell == cell && zi == iadd(icell, 1)) ? 1 : 0;
        cell = zs;
        icell = zi;
        return from;
    }
};

// Lattice cell and offsets of the fixed axes (recomputed at each rebuild: cheaper than the
// registers that would hold them).
template <int D>
FND void col_lattice(const float* q, int (*c)[2], float (*f)[2])
{
#pragma unroll
    for (int k = 0; k < D - 1; ++k) {
        const float fl = floorf(q[k]);
        c[k][0] = imul(cvti(fl), kPrimes[k]);
        c[k][1] = iadd(c[k][0], kPrimes[k]);
        f[k][0] = q[k] - fl;
        f[k][1] = f[k][0] - 1.0f;
    }
}

// `pos(q)` writes the D - 1 fixed coordinates (already scaled by the node's frequency).
// The lower and the upper lattice plane run as the two halves of packed operations (256^3
// FBm(Perlin): 142 us; scalar operations 151 us; the point kernel 515 us).  The rebuild loop
// works on scalars and packs at its end: kept pairs updated half by half inside the loop came
// out of the compiler with both halves new (tests/test_gpu_column.py would show it).
template <int D>
struct PerlinCol {
    static constexpr int N = 1 << (D - 1);        // corners of one lattice plane
    f32x2 s[N], g[N];                             // (lower, upper) plane: dot = fma(s, t, g)
    float ease[D - 1];
    ColCell at;

    template <typename Pos>
    FND void init(Pos&& pos)
    {
        float q[D - 1];
        pos(q);
#pragma unroll
        for (int k = 0; k < D - 1; ++k) ease[k] = quintic(q[k] - floorf(q[k]));
#pragma unroll
        for (int m = 0; m < N; ++m) s[m] = g[m] = 0;
        at.init();
    }
    FND unsigned prepare(float4* tab, unsigned lane, float Z)
    {
        return at.prepare(tab, lane, Z, [](float t) { return quintic(t); });
    }
    template <typename Pos>
    FND void enter(int seed, float zs, Pos&& pos)
    {
        if (zs != at.cell) {
            int zi;
            float q[D - 1], f[D - 1][2];
            int c[D - 1][2];
            pos(q);
            col_lattice<D>(q, c, f);
            float ls[N], lg[N], hs[N], hg[N];
#pragma unroll
            for (int m = 0; m < N; ++m) {
                unpack2(s[m], ls[m], hs[m]);
                unpack2(g[m], lg[m], hg[m]);
            }
#pragma unroll 1
            for (int k = at.enter(zs, zi); k < 2; ++k) {
                const int zh = seed ^ imul(iadd(zi, k), kPrimes[D - 1]);
#pragma unroll
                for (int m = 0; m < N; ++m) {
                    const int b0 = m & 1, b1 = (m >> 1) & 1, b2 = (m >> 2) & 1;
                    int h = zh ^ c[0][b0] ^ c[1][b1];
                    if constexpr (D == 4) h ^= c[2 % (D - 1)][b2];
                    h = hash_mix(h);
                    ls[m] = hs[m];
                    lg[m] = hg[m];
                    if constexpr (D == 3) grad_col3(h, f[0][b0], f[1][b1], hs[m], hg[m]);
                    else grad_col4(h, f[0][b0], f[1][b1], f[2 % (D - 1)][b2], hs[m], hg[m]);
                }
            }
#pragma unroll
            for (int m = 0; m < N; ++m) {
                s[m] = pack2(ls[m], hs[m]);
                g[m] = pack2(lg[m], hg[m]);
            }
        }
    }
    FND float eval(const float4& e) const
    {
        const f32x2 z = pack2(e.x, e.y);
        f32x2 v[N];
#pragma unroll
        for (int m = 0; m < N; ++m) v[m] = fma2(s[m], z, g[m]);
#pragma unroll
        for (int k = 0; k < D - 1; ++k) {
            const f32x2 t = pack2(ease[k], ease[k]);
#pragma unroll
            for (int j = 0; j < (N >> (k + 1)); ++j) v[j] = lerp2(v[2 * j], v[2 * j + 1], t);
        }
        float lo, hi;
        unpack2(v[0], lo, hi);
        return lerp(lo, hi, e.z);
    }
};

// 2D: dot = fma(1 + sqrt 2, a, b) with (a, b) the signed offsets, in either order; the one
// along the column is p * t, the other is kept (q), so a = fma(pa, t, qa), b = fma(pb, t, qb)
// with one of each pair zero.
template <>
struct PerlinCol<2> {
    float pa[2][2], qa[2][2], pb[2][2], qb[2][2];   // [plane][x corner]
    float ease;
    ColCell at;

    template <typename Pos>
    FND void init(Pos&& pos)
    {
        float q[1];
        pos(q);
        ease = quintic(q[0] - floorf(q[0]));
#pragma unroll
        for (int m = 0; m < 4; ++m) pa[m >> 1][m & 1] = qa[m >> 1][m & 1] = pb[m >> 1][m & 1] = qb[m >> 1][m & 1] = 0.0f;
        at.init();
    }
    FND unsigned prepare(float4* tab, unsigned lane, float Y)
    {
        return at.prepare(tab, lane, Y, [](float t) { return quintic(t); });
    }
    template <typename Pos>
    FND void enter(int seed, float ys, Pos&& pos)
    {
        if (ys != at.cell) {
            int yi;
            float q[1], f[1][2];
            int c[1][2];
            pos(q);
            col_lattice<2>(q, c, f);
#pragma unroll 1
            for (int k = at.enter(ys, yi); k < 2; ++k) {
                const int yh = seed ^ imul(iadd(yi, k), kPrimeY);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    pa[0][m] = pa[1][m]; qa[0][m] = qa[1][m]; pb[0][m] = pb[1][m]; qb[0][m] = qb[1][m];
                    const int h = hash_mix(yh ^ c[0][m]);
                    const bool swap = (h << 29) < 0;
                    const float xv = flip(f[0][m], h << 31), sy = flip(1.0f, h << 30);
                    pa[1][m] = swap ? sy : 0.0f;
                    qa[1][m] = swap ? 0.0f : xv;
                    pb[1][m] = swap ? 0.0f : sy;
                    qb[1][m] = swap ? xv : 0.0f;
                }
            }
        }
    }
    FND float eval(const float4& e) const
    {
        float d[2][2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const float t = k ? e.y : e.x;
                d[k][m] = fmaf(1.0f + (float)kRoot2, fmaf(pa[k][m], t, qa[k][m]), fmaf(pb[k][m], t, qb[k][m]));
            }
        return lerp(lerp(d[0][0], d[0][1], ease), lerp(d[1][0], d[1][1], ease), e.z);
    }
};

// Value noise: a lattice plane interpolated across the fixed axes is one number; a step is
// the easing curve and the last lerp.
template <int D>
struct ValueCol {
    static constexpr int N = 1 << (D - 1);
    float lo, hi;
    ColCell at;

    template <typename Pos>
    FND void init(Pos&&) { lo = hi = 0.0f; at.init(); }
    FND unsigned prepare(float4* tab, unsigned lane, float Z)
    {
        return at.prepare(tab, lane, Z, [](float t) { return hermite(t); });
    }
    template <typename Pos>
    FND void enter(int seed, float zs, Pos&& pos)
    {
        if (zs != at.cell) {
            int zi;
            float q[D - 1], f[D - 1][2];
            int c[D - 1][2];
            pos(q);
            col_lattice<D>(q, c, f);
#pragma unroll 1
            for (int k = at.enter(zs, zi); k < 2; ++k) {
                const int zh = seed ^ imul(iadd(zi, k), kPrimes[D - 1]);
                float v[N];
#pragma unroll
                for (int m = 0; m < N; ++m) {
                    int h = zh ^ c[0][m & 1];
                    if constexpr (D >= 3) h ^= c[1 % (D - 1)][(m >> 1) & 1];
                    if constexpr (D == 4) h ^= c[2 % (D - 1)][(m >> 2) & 1];
                    v[m] = valcoord(h);
                }
#pragma unroll
                for (int a = 0; a < D - 1; ++a)
#pragma unroll
                    for (int j = 0; j < (N >> (a + 1)); ++j) v[j] = lerp(v[2 * j], v[2 * j + 1], hermite(f[a][0]));
                lo = hi;
                hi = v[0];
            }
        }
    }
    FND float eval(const float4& e) const { return lerp(lo, hi, e.z); }
};

// Cellular noise with a constant jitter and (squared) Euclidean distance, 2D and 3D.  A
// step's 3^D cells are the same while the column stays in its cell: the warp computes the
// jittered points of each distinct cell neighbourhood its lanes need (one lane per cell) into
// shared memory, and every lane keeps each cell's squared distance across the column, so a
// step is two fmas per cell, packed for pairs of cells, and a comparison, in the reference's
// order, without pruning (CellularLookup 160^3 48.6 us with scalar fmas, 44.9 us packed; the
// compares' half-rate pipe and the short columns' set-up bound it now).
// Neighbourhoods beyond kGroups per warp and positions past 1e9 (or NaN) take the point
// function; `fast` says which, the same for all lanes.
enum ColCellKind { kColValue, kColDistance, kColLookup };

template <int D, ColCellKind Kind, int NS = 1>
struct CellCol {
    static constexpr int N = D == 3 ? 27 : 9, kGroups = 4;
    static constexpr int M = N / 3, MP = D == 3 ? 12 : 4;   // cells of one plane across the column, padded
    f32x2 part[3][(M + 1) / 2];                   // squared distance across the column, cells of a plane in pairs
    int icell;
    unsigned slot;                                // this lane's neighbourhood in the table
    bool fast;

    // per warp behind the 32 step entries: kGroups x N cells (direction and scale, or the cell
    // point for kColLookup); per group and plane what a step reads, as arrays over the plane's
    // cells (the column components, then the scales); the hashes (kColValue)
    static constexpr int kAlong = Kind == kColLookup ? MP : 2 * MP;          // floats per plane
    static constexpr int kTable = 32 + kGroups * N + kGroups * 3 * kAlong / 4 + (Kind == kColValue ? N : 0);
    static FND const float* along(const float4* tab, unsigned slot, int plane)
    {
        return reinterpret_cast<const float*>(tab + 32 + kGroups * N) + (slot * 3u + plane) * kAlong;
    }
    static FND int* hashes(float4* tab) { return reinterpret_cast<int*>(tab + 32 + kGroups * N + kGroups * 3 * kAlong / 4); }

    template <typename Pos>
    FND void init(Pos&&)
    {
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < (M + 1) / 2; ++j) part[k][j] = 0;
        icell = 0x7fffffff;
        slot = 0;
        fast = false;
    }
    // entry: the column offsets of the three cell planes as the walk of this kind computes them
    // (kColLookup: the coordinate), and the plane's base cell (INT_MIN: no fast cell)
    FND unsigned prepare(float4* tab, unsigned lane, float p)
    {
        const int base = fabs_(p) < 1e9f ? iadd(cvti(p), -1) : (int)0x80000000;
        const float c0 = cvtf(base), c1 = c0 + 1.0f, c2 = c1 + 1.0f;
        float4 e;
        if (Kind == kColValue) { e.x = c0 - p; e.y = e.x + 1.0f; e.z = e.y + 1.0f; }
        else if (Kind == kColDistance) { e.x = c0 - p; e.y = c1 - p; e.z = c2 - p; }
        else { e.x = e.y = e.z = p; }
        e.w = __int_as_float(base);
        tab[lane] = e;
        const int before = __shfl_up_sync(0xffffffffu, base, 1);
        return __ballot_sync(0xffffffffu, base != (lane ? before : icell));
    }
    template <typename Pos>
    FND void enter(int seed, float4* tab, unsigned j, float jitter, Pos&& pos)
    {
        const int base = __float_as_int(tab[j].w);
        if (base == icell) return;
        icell = base;
        float q[D - 1];
        int cb[D - 1];
        pos(q);
        bool sane = base != (int)0x80000000;
#pragma unroll
        for (int k = 0; k < D - 1; ++k) {
            sane = sane && fabs_(q[k]) < 1e9f;
            cb[k] = iadd(cvti(q[k]), -1);
        }
        fast = __all_sync(0xffffffffu, sane) != 0;
        if (!fast) return;
        float4* cells = tab + 32;
        const int lane = (int)(threadIdx.x & 31u);
        const int at[3] = {D == 3 ? lane / 9 : lane / 3, D == 3 ? (lane / 3) % 3 : lane % 3, lane % 3};
        unsigned todo = 0xffffffffu, groups = 0;
        __syncwarp();
#pragma unroll 1
        do {
            const int leader = __ffs((int)todo) - 1;
            int c[D];
            float cf[D];
            bool mine = true;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int b = k == D - 1 ? base : __shfl_sync(0xffffffffu, cb[k % (D - 1)], leader);
                if (k < D - 1) mine = mine && cb[k % (D - 1)] == b;
                c[k] = imul(iadd(b, at[k]), kPrimes[k]);
                cf[k] = cvtf(b);
                if (at[k] > 0) cf[k] += 1.0f;
                if (at[k] > 1) cf[k] += 1.0f;
            }
            if (lane < N) {
                const int h = cell_hash<D>(seed, c);
                float d[D + 1];
                cell_dir_raw<D>(h, d);
                cell_dir_scale<D>(jitter, d);
                float4 e;
                if (Kind == kColLookup) {
                    e.x = fmaf(d[0], d[D], cf[0]);
                    e.y = fmaf(d[1], d[D], cf[1]);
                    e.z = D == 3 ? fmaf(d[2 % D], d[D], cf[2 % D]) : 0.0f;
                    e.w = 0.0f;
                } else {
                    e = D == 3 ? make_float4(d[0], d[1], d[2 % D], d[D]) : make_float4(d[0], 0.0f, d[1], d[D]);
                }
                cells[groups * N + lane] = e;
                // lane = 3 m + plane
                float* a = const_cast<float*>(along(tab, groups, lane % 3)) + lane / 3;
                if (Kind == kColLookup) {
                    a[0] = D == 3 ? e.z : e.y;
                } else {
                    a[0] = e.z;
                    a[MP] = e.w;
                }
                if (Kind == kColValue) hashes(tab)[groups * N + lane] = h;
            }
            if (mine) slot = groups;
            todo &= ~__ballot_sync(0xffffffffu, mine);
            ++groups;
        } while (todo && groups < (unsigned)kGroups);
        __syncwarp();
        fast = todo == 0;
        if (!fast) return;
        float t[D - 1][3];
#pragma unroll
        for (int k = 0; k < D - 1; ++k) {
            const float c0 = cvtf(cb[k]), c1 = c0 + 1.0f, c2 = c1 + 1.0f;
            t[k][0] = c0 - q[k];
            t[k][1] = Kind == kColValue ? t[k][0] + 1.0f : c1 - q[k];
            t[k][2] = Kind == kColValue ? t[k][1] + 1.0f : c2 - q[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int m = 0; m < M; m += 2) {
                float d[2] = {0.0f, 0.0f};
#pragma unroll
                for (int h = 0; h < 2 && m + h < M; ++h) {
                    const float4 e = cells[slot * N + (m + h) * 3 + k];
                    const int i0 = D == 3 ? (m + h) / 3 : m + h, i1 = (m + h) % 3;
                    const float o0 = Kind == kColLookup ? e.x - q[0] : fmaf(e.x, e.w, t[0][i0]);
                    d[h] = o0 * o0;
                    if (D == 3) {
                        const float o1 = Kind == kColLookup ? e.y - q[1 % (D - 1)] : fmaf(e.y, e.w, t[1 % (D - 1)][i1]);
                        d[h] = fmaf(o1, o1, d[h]);
                    }
                }
                part[k][m / 2] = pack2(d[0], d[1]);
            }
    }
    // squared distances at a step, two cells of a plane at a time (plane k, cells 2 j, 2 j + 1)
    FND void dist2(const float4* tab, unsigned j, float (*d)[M + 1]) const
    {
        const float4 e = tab[j];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float* a = along(tab, slot, k);
            const float t = k == 0 ? e.x : (k == 1 ? e.y : e.z);
            const f32x2 tt = pack2(t, t);
#pragma unroll
            for (int m = 0; m < M; m += 4) {
                const float4 z = *reinterpret_cast<const float4*>(a + m);
                float4 w;
                if (Kind != kColLookup) w = *reinterpret_cast<const float4*>(a + MP + m);
#pragma unroll
                for (int h = 0; h < 4 && m + h < M; h += 2) {
                    const f32x2 zz = h ? pack2(z.z, z.w) : pack2(z.x, z.y);
                    const f32x2 o = Kind == kColLookup ? sub2(zz, tt) : fma2(zz, h ? pack2(w.z, w.w) : pack2(w.x, w.y), tt);
                    unpack2(fma2(o, o, part[k][(m + h) / 2]), d[k][m + h], d[k][m + h + 1]);
                }
            }
        }
    }
    // index of the closest cell, the first of equals
    FND int closest(const float4* tab, unsigned j) const
    {
        float d[3][M + 1];
        dist2(tab, j, d);
        float best = d[0][0];
        int at = 0;
#pragma unroll
        for (int i = 1; i < N; ++i) {
            const float v = d[i % 3][i / 3];
            at = v < best ? i : at;
            best = fminf(best, v);                // finite: the same as a select, off the half-rate compares
        }
        return at;
    }
    FND float value(const float4* tab, unsigned j) const
    {
        return cvtf(hashes(const_cast<float4*>(tab))[slot * N + closest(tab, j)]);
    }
    FND void distances(const float4* tab, unsigned j, float* dist) const
    {
        float v[3][M + 1];
        dist2(tab, j, v);
        dist[0] = dist[1] = dist[2] = dist[3] = __int_as_float(0x7F800000);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float d = v[i % 3][i / 3];
            if (NS > 1) dist[1] = fmaxf(fminf(dist[1], d), dist[0]);
            dist[0] = fminf(dist[0], d);
        }
    }
    FND void lookup(const float4* tab, unsigned j, float scale, float* out) const
    {
        const float4 e = tab[32 + slot * N + closest(tab, j)];
        out[0] = e.x * scale;
        out[1] = e.y * scale;
        if (D == 3) out[2 % D] = e.z * scale;
    }
};

// DomainWarpGradient at a separable position, 2D and 3D: the corner vectors of the lattice cell
// are the same while the column stays in it.  The warp keeps those of each distinct cell of its
// lanes in shared memory (converted, one lane per corner), a lane its corners' weights across
// the column; a step is one broadcast load and a packed and a scalar fma per corner (46
// instructions in 3D against ~150 with hashing and conversions).  More than kGroups cells per
// warp take the point function (`fast`).
template <int D>
struct WarpCol {
    static constexpr int N = 1 << D, kGroups = 4, kTable = 32 + kGroups * N;
    float weight[N / 2];                          // of the corners across the column
    int icell;
    unsigned slot;
    bool fast;

    template <typename Pos>
    FND void init(Pos&& pos)
    {
        float q[D - 1], s[2][2];
        pos(q);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            s[k][1] = hermite(q[k % (D - 1)] - floorf(q[k % (D - 1)]));
            s[k][0] = 1.0f - s[k][1];
        }
#pragma unroll
        for (int m = 0; m < N / 2; ++m) weight[m] = D == 2 ? s[0][m] : s[0][m & 1] * s[1][m >> 1];
        icell = 0x7fffffff;
        slot = 0;
        fast = false;
    }
    // entry: weights of the lower and the upper plane, -, the cell
    FND unsigned prepare(float4* tab, unsigned lane, float p)
    {
        const float fl = floorf(p), s1 = hermite(p - fl);
        const int cell = cvti(fl);
        tab[lane] = make_float4(1.0f - s1, s1, 0.0f, __int_as_float(cell));
        const int before = __shfl_up_sync(0xffffffffu, cell, 1);
        return __ballot_sync(0xffffffffu, cell != (lane ? before : icell));
    }
    template <typename Pos>
    FND void enter(int seed, float4* tab, unsigned j, float, Pos&& pos)
    {
        const int cell = __float_as_int(tab[j].w);
        if (cell == icell) return;
        icell = cell;
        float q[D - 1];
        int cb[D - 1];
        pos(q);
#pragma unroll
        for (int k = 0; k < D - 1; ++k) cb[k] = cvti(floorf(q[k]));
        const int lane = (int)(threadIdx.x & 31u);
        unsigned todo = 0xffffffffu, groups = 0;
        __syncwarp();
#pragma unroll 1
        do {
            const int leader = __ffs((int)todo) - 1;
            int c[D];
            bool mine = true;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int b = k == D - 1 ? cell : __shfl_sync(0xffffffffu, cb[k % (D - 1)], leader);
                if (k < D - 1) mine = mine && cb[k % (D - 1)] == b;
                c[k] = imul(iadd(b, (lane >> k) & 1), kPrimes[k]);
            }
            if (lane < N) {
                const int h = cell_hash<D>(seed, c);
                tab[32 + groups * N + lane] = D == 2 ? make_float4(cvtf(h & 0xffff), cvtf((int)srl(h, 16)), 0.0f, 0.0f)
                                                     : make_float4(cvtf(h & 0x3ff), cvtf((h >> 11) & 0x3ff), cvtf((int)srl(h, 22)), 0.0f);
            }
            if (mine) slot = groups * N;
            todo &= ~__ballot_sync(0xffffffffu, mine);
            ++groups;
        } while (todo && groups < (unsigned)kGroups);
        __syncwarp();
        fast = todo == 0;
    }
    FND float warp(const float4* tab, unsigned j, float amp, const float* axis, float* io) const
    {
        const float4 e = tab[j];
        const float4* corners = tab + 32 + slot;
        f32x2 v01 = 0;
        float wv[D];
#pragma unroll
        for (int m = 0; m < N; ++m) {
            const float4 c = corners[m];
            const float t = weight[m & (N / 2 - 1)] * (m < N / 2 ? e.x : e.y);
            const f32x2 tt = pack2(t, t), c01 = pack2(c.x, c.y);
            v01 = m == 0 ? mul2(tt, c01) : fma2(tt, c01, v01);
            if (D == 3) wv[2 % D] = m == 0 ? t * c.z : fmaf(t, c.z, wv[2 % D]);
        }
        unpack2(v01, wv[0], wv[1]);
        constexpr float normalise = D == 2 ? 1.0f / (0xffff / 2.0f) : 1.0f / (0x3ff / 2.0f);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            wv[k] = fmaf(wv[k], normalise, -1.0f);
            io[k] = fmaf(wv[k], amp * axis[k], io[k]);
        }
        float r = wv[D - 1] * wv[D - 1];
#pragma unroll
        for (int k = D - 2; k >= 0; --k) r = fmaf(wv[k], wv[k], r);
        return r;
    }
};

}  // namespace fnd
