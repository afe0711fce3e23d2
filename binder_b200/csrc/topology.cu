// Jacobian determinants and topology correction in FP64.
//
// This file is compiled with -fmad=false: every determinant is evaluated with the reference's
// expression grouping and without fused multiply-adds, so the per-voxel Jacobians (and therefore
// the negative / out-of-range counts and the set of corners the limiter touches) equal the
// reference CPU backend's bit for bit on the same FP64 input.
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "layout.cuh"
#include "hartley.cuh"
#include "topology.cuh"

namespace binder {

namespace {

// cofactor expansion along the first row with the reference's grouping
// (BINDER/src/cpu/utils.cpp:156-160, topology_correction_3D.cpp:286-288)
__device__ __forceinline__ double det3(double a00, double a01, double a02, double a10, double a11,
                                       double a12, double a20, double a21, double a22) {
    return a00 * (a11 * a22 - a12 * a21) - a01 * (a10 * a22 - a12 * a20) +
           a02 * (a10 * a21 - a11 * a20);
}

__device__ __forceinline__ unsigned long long ordered(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
double unordered(unsigned long long o) {
    const unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    double v;
    memcpy(&v, &b, sizeof(v));
    return v;
}

struct Red {
    unsigned long long mn, mx;
    unsigned long long below, above, negative;
    double sum[3];
    int pad;
};

// BINDER/src/cpu/utils.cpp:100-345.  Element (p, m) of the field is f[p*ps + m*cs].  Four corners
// share each difference; bound by the FP64 pipe.  160x192x160: 164 us with the differences taken
// per corner, 97 us so.
__global__ void jacobian_kernel(const double *f, long ps, long cs, int nx, int ny, int nz,
                                double vol, double *J, double e1, double e2, Red *red) {
    const long V = (long)nx * ny * nz;
    const long yz = (long)ny * nz;
    // corner order of the reference: fff, bff, fbf, ffb, bbf, bfb, fbb, bbb
    constexpr int dir[8][3] = {{1, 1, 1},  {-1, 1, 1},  {1, -1, 1},  {1, 1, -1},
                           {-1, -1, 1}, {-1, 1, -1}, {1, -1, -1}, {-1, -1, -1}};
    double lmin = 1e300, lmax = -1e300;
    unsigned long long lb = 0, la = 0, ln = 0;
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x) {
        int x, y, z;
        if (V <= 0xffffffffL) {  // 32-bit divisions
            const unsigned q = (unsigned)p, row = q / (unsigned)nz;
            z = (int)(q - row * nz);
            x = (int)(row / (unsigned)ny);
            y = (int)(row - (unsigned)x * ny);
        } else {
            x = (int)(p / yz), y = (int)((p / nz) % ny), z = (int)(p % nz);
        }
        // the differences to the next (0) and from the previous (1) point along each axis, where
        // there is one (the point itself stands in where there is none)
        const bool ok[3][2] = {{x < nx - 1, x > 0}, {y < ny - 1, y > 0}, {z < nz - 1, z > 0}};
        const long step[3] = {yz, nz, 1};
        double d[3][2][3];  // [axis][side][component]
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const double w0 = f[p * ps + m * cs];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                d[a][0][m] = f[(ok[a][0] ? p + step[a] : p) * ps + m * cs] - w0;
                d[a][1][m] = w0 - f[(ok[a][1] ? p - step[a] : p) * ps + m * cs];
            }
        }
        double tot = 0.0;
        int valid = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int sx = dir[c][0] < 0, sy = dir[c][1] < 0, sz = dir[c][2] < 0;
            if (!(ok[0][sx] && ok[1][sy] && ok[2][sz])) continue;
            const double *u = d[0][sx], *v = d[1][sy], *w = d[2][sz];
            const double jc = det3(u[0], v[0], w[0], u[1], v[1], w[1], u[2], v[2], w[2]) * vol;
            tot += jc;
            valid++;
        }
        const double jv = valid > 0 ? tot / valid : 1.0;
        if (J) J[p] = jv;
        lmin = fmin(lmin, jv);
        lmax = fmax(lmax, jv);
        lb += jv < e1;
        la += jv > e2;
        ln += jv < 0.0;
    }
    if (red) {
        // warp-level first, then one atomic per warp
        for (int o = 16; o > 0; o >>= 1) {
            lmin = fmin(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
            lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
            lb += __shfl_xor_sync(0xffffffffu, lb, o);
            la += __shfl_xor_sync(0xffffffffu, la, o);
            ln += __shfl_xor_sync(0xffffffffu, ln, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&red->mn, ordered(lmin));
            atomicMax(&red->mx, ordered(lmax));
            if (lb) atomicAdd(&red->below, lb);
            if (la) atomicAdd(&red->above, la);
            if (ln) atomicAdd(&red->negative, ln);
        }
    }
}

// BINDER/src/cpu/utils.cpp:10-98: the 2D Jacobian averaged over the 4 one-sided corners (orders
// fxfy, bxfy, fxby, bxby), each the determinant of the forward / backward differences, with the
// reference's expression grouping.  Element (p, m) of the field is f[p*ps + m*cs]; J and red are
// optional, as in jacobian_kernel.
__global__ void jacobian2d_kernel(const double *f, long ps, long cs, int nx, int ny, double vol,
                                  double *J, double e1, double e2, Red *red) {
    const long V = (long)nx * ny;
    const int dir[4][2] = {{1, 1}, {-1, 1}, {1, -1}, {-1, -1}};
    double lmin = 1e300, lmax = -1e300;
    unsigned long long lb = 0, la = 0, ln = 0;
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x) {
        const int x = (int)(p / ny), y = (int)(p % ny);
        const double w0 = f[p * ps], w1 = f[p * ps + cs];
        double tot = 0.0;
        int valid = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int sx = dir[c][0], sy = dir[c][1];
            if ((sx > 0 && x >= nx - 1) || (sx < 0 && x <= 0)) continue;
            if ((sy > 0 && y >= ny - 1) || (sy < 0 && y <= 0)) continue;
            const long qx = p + (long)sx * ny, qy = p + sy;
            const double bx0 = f[qx * ps], bx1 = f[qx * ps + cs];
            const double by0 = f[qy * ps], by1 = f[qy * ps + cs];
            const double ax0 = sx > 0 ? bx0 - w0 : w0 - bx0;
            const double ax1 = sx > 0 ? bx1 - w1 : w1 - bx1;
            const double ay0 = sy > 0 ? by0 - w0 : w0 - by0;
            const double ay1 = sy > 0 ? by1 - w1 : w1 - by1;
            tot += (ax0 * ay1 - ay0 * ax1) * vol;
            valid++;
        }
        const double jv = valid > 0 ? tot / valid : 1.0;
        if (J) J[p] = jv;
        lmin = fmin(lmin, jv);
        lmax = fmax(lmax, jv);
        lb += jv < e1;
        la += jv > e2;
        ln += jv < 0.0;
    }
    if (red) {
        for (int o = 16; o > 0; o >>= 1) {
            lmin = fmin(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
            lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
            lb += __shfl_xor_sync(0xffffffffu, lb, o);
            la += __shfl_xor_sync(0xffffffffu, la, o);
            ln += __shfl_xor_sync(0xffffffffu, ln, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&red->mn, ordered(lmin));
            atomicMax(&red->mx, ordered(lmax));
            if (lb) atomicAdd(&red->below, lb);
            if (la) atomicAdd(&red->above, la);
            if (ln) atomicAdd(&red->negative, ln);
        }
    }
}

// topology_correction_3D.cpp:488-607: the 8 vertex Jacobians of every cell, in the vertex order
// 000, 100, 010, 001, 011, 101, 110, 111, each from the three cell edges through its vertex.
// Positions are SoA [3][V].  The limiter asks only which of them lie outside [e1, e2]: bit c of
// mask[cell] (storing the eight values moved 64 B per cell and took twice as long).  The two corners of
// an edge share its difference, and V <= 2^24 keeps the indices in 32 bits.  Bound by the FP64 pipe.
// 160x192x160: 110 us with an edge per corner and 64-bit indices, 88 us so.
__global__ void corner_kernel(const double *pos, int nx, int ny, int nz, double vol, double e1,
                              double e2, uint8_t *mask, Red *red) {
    const unsigned V = (unsigned)nx * ny * nz, cy = ny - 1, cz = nz - 1;
    const unsigned cells = (unsigned)(nx - 1) * cy * cz;
    constexpr int vert[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1},
                                {0, 1, 1}, {1, 0, 1}, {1, 1, 0}, {1, 1, 1}};
    unsigned long long lb = 0, la = 0;
    for (unsigned cell = blockIdx.x * blockDim.x + threadIdx.x; cell < cells;
         cell += gridDim.x * blockDim.x) {
        const unsigned row = cell / cz, z = cell - row * cz, x = row / cy, y = row - x * cy;
        const double *node = pos + ((size_t)(x * ny + y) * nz + z);
        // the cell's edges along each axis, [the two other coordinates][component], far end minus
        // near end: two corners share each
        double ex[4][3], ey[4][3], ez[4][3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            double p[2][2][2];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        p[a][b][c] = node[(size_t)m * V + (unsigned)((a * ny + b) * nz + c)];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    ex[2 * a + b][m] = p[1][a][b] - p[0][a][b];
                    ey[2 * a + b][m] = p[a][1][b] - p[a][0][b];
                    ez[2 * a + b][m] = p[a][b][1] - p[a][b][0];
                }
        }
        unsigned bits = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const double *u = ex[2 * vert[c][1] + vert[c][2]], *v = ey[2 * vert[c][0] + vert[c][2]],
                         *w = ez[2 * vert[c][0] + vert[c][1]];
            double j = det3(u[0], v[0], w[0], u[1], v[1], w[1], u[2], v[2], w[2]);
            j *= vol;
            lb += j < e1;
            la += j > e2;
            bits |= (j < e1 || j > e2) ? 1u << c : 0u;
        }
        mask[cell] = (uint8_t)bits;
    }
    for (int o = 16; o > 0; o >>= 1) {
        lb += __shfl_xor_sync(0xffffffffu, lb, o);
        la += __shfl_xor_sync(0xffffffffu, la, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (lb) atomicAdd(&red->below, lb);
        if (la) atomicAdd(&red->above, la);
    }
}

// red->sum[n] += the CTA's s[n]; every thread of the CTA
template <int N>
__device__ __forceinline__ void add_sums(double (&s)[N], Red *red) {
    __shared__ double part[32];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const double v = block_sum(s[n], part);
        if (threadIdx.x == 0) atomicAdd(&red->sum[n], v);
    }
}

// topology_correction_3D.cpp:172-245: periodic forward differences, g[(n1*3+n2)][p] =
// (pos_n1(p + e_n2) - pos_n1(p)) / vs[n1], and the sums of the positions into red.  32-bit indices
// (V <= 2^24).  EXACT: every vs is a power of two, so the products with the reciprocals (v0 .. v2) are
// the quotients to the bit.  Bound by DRAM, with the nine FP64 divisions a voxel by those.
// 160x192x160: 126 us with 64-bit indices, and 71 for the sums in a kernel of their own; now 121
// together, 85 without the divisions.
template <bool EXACT>
__global__ void gradient_kernel(const double *pos, int nx, int ny, int nz, double v0, double v1,
                                double v2, double *g, Red *red) {
    const unsigned V = (unsigned)nx * ny * nz;
    const double vs[3] = {v0, v1, v2};
    double s[3] = {0.0, 0.0, 0.0};
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < V; p += gridDim.x * blockDim.x) {
        const unsigned row = p / nz, z = p - row * nz, x = row / ny, y = row - x * ny;
        const unsigned px = x + 1 == (unsigned)nx ? p - (nx - 1) * ny * nz : p + ny * nz;
        const unsigned py = y + 1 == (unsigned)ny ? p - (ny - 1) * nz : p + nz;
        const unsigned pz = z + 1 == (unsigned)nz ? p - (nz - 1) : p + 1;
#pragma unroll
        for (int n1 = 0; n1 < 3; ++n1) {
            const double *f = pos + (size_t)n1 * V;
            double *o = g + (size_t)n1 * 3 * V + p;
            const double c = f[p];
            s[n1] += c;
            o[0] = EXACT ? (f[px] - c) * vs[n1] : (f[px] - c) / vs[n1];
            o[V] = EXACT ? (f[py] - c) * vs[n1] : (f[py] - c) / vs[n1];
            o[2 * (size_t)V] = EXACT ? (f[pz] - c) * vs[n1] : (f[pz] - c) / vs[n1];
        }
    }
    add_sums(s, red);
}

template <int N>
__device__ __forceinline__ double detn(const double (&J)[N][N]) {
    if constexpr (N == 2)
        return J[0][0] * J[1][1] - J[0][1] * J[1][0];
    else
        return det3(J[0][0], J[0][1], J[0][2], J[1][0], J[1][1], J[1][2], J[2][0], J[2][1], J[2][2]);
}

// topology_correction_3D.cpp:247-332 and topology_correction_2D.cpp:248-313.  The reference visits
// cells in lexicographic order and a cell's corners in order; a cell reads and writes gradients only
// inside its 2x2x2 (2x2) footprint, so two cells interact only if they differ by at most 1 along
// every axis.  A flagged cell may therefore go as soon as its flagged neighbours that come before it
// have gone: cells with none go first (round 0), and each cell counts down its later neighbours, the
// last count putting one into the next round.  The cells of a round are no neighbours of each other,
// so the result is the sequential walk's exactly, and the rounds are as many as the longest chain of
// neighbouring cells: 42 for a 160x192x160 field with 157,751 flagged cells, 58 for a 128x128 one
// with 2,253.
//
// A step: J is a corner's matrix of gradients, replaced by (1 - alpha) J + alpha I.  The reference
// steps alpha by 0.1 (capped at 1) until det((1 - alpha) J + alpha I) lies in [e1, e2], at most 11
// steps from 0, then takes one step more.  The alphas are constants, so the trials are independent:
// four lanes share a cell and try four alphas at a time, and the lowest trial in range picks the
// step.  The field's values of a cell stay in shared memory from its first corner to its last.
// FP64 work and the chain of a cell's corners bound it: with 16 lanes to a cell, all twelve trials
// at once and the values passed around by shuffles, one CTA took 153 us where this takes 138
// (22x24x24, 6,517 flagged cells, 130 rounds); a wavefront over the levels 2x + y of an image took
// 130 us where the rounds take 38 (128x128).
struct LimiterArgs {
    const uint8_t *mask;  // flagged corners of every cell (corner_kernel, corner2d_kernel)
    double *g;            // gradients [N * N][V]
    int *deg;             // earlier flagged neighbours still to go, per cell
    int *front[2];        // the cells of a round and of the next
    int *counts;          // cells of each round
    int nx, ny, nz;       // nz = 1: an image
    double e1, e2;
    unsigned *flags;
};

constexpr int kTrials = 12;  // alphas of 0 .. 11 steps
// al[k]: alpha after k steps, k <= kTrials
__device__ __forceinline__ void step_alphas(double *al) {
    double a = 0.0;
    for (int k = 0; k <= kTrials; ++k) {
        al[k] = a;
        a = a + 0.1;
        if (a > 1.0) a = 1.0;
    }
}

// a grid of cells: how a flat index, the later neighbours and a cell's values are laid out
template <int DIM>
struct CellGrid {
    static constexpr int kLater = DIM == 3 ? 13 : 4;    // later neighbours in lexicographic order
    static constexpr int kPerLane = DIM == 3 ? 9 : 2;   // of the 36 (8) values, by 4 lanes
    static constexpr int kStride = 4 * kPerLane + 1;    // doubles of scratch per cell
    int cx, cy, cz;
    __device__ __forceinline__ explicit CellGrid(const LimiterArgs &a)
        : cx(a.nx - 1), cy(a.ny - 1), cz(DIM == 3 ? a.nz - 1 : 1) {}
    __device__ __forceinline__ int count() const { return cx * cy * cz; }
    __device__ __forceinline__ void at(int cell, int &x, int &y, int &z) const {
        const int row = DIM == 3 ? cell / cz : cell;
        z = DIM == 3 ? cell - row * cz : 0;
        x = row / cy;
        y = row - x * cy;
    }
    // the later neighbour q of (x, y, z), or the earlier one with sign -1; -1 outside
    __device__ __forceinline__ int neighbour(int q, int sign, int x, int y, int z) const {
        const int o = q + kLater + 1;  // 27 (9) offsets in order, the cell itself in the middle
        const int X = x + sign * (DIM == 3 ? o / 9 - 1 : o / 3 - 1);
        const int Y = y + sign * (DIM == 3 ? o / 3 % 3 - 1 : o % 3 - 1);
        const int Z = DIM == 3 ? z + sign * (o % 3 - 1) : 0;
        const bool in = (unsigned)X < (unsigned)cx && (unsigned)Y < (unsigned)cy &&
                        (DIM == 2 || (unsigned)Z < (unsigned)cz);
        return in ? (X * cy + Y) * cz + Z : -1;
    }
    // earlier flagged neighbours of a flagged cell
    __device__ __forceinline__ int earlier_flagged(const uint8_t *mask, int cell) const {
        int x, y, z, n = 0;
        at(cell, x, y, z);
#pragma unroll
        for (int q = 0; q < kLater; ++q) {
            const int nb = neighbour(q, -1, x, y, z);
            if (nb >= 0) n += mask[nb] != 0;
        }
        return n;
    }
};

// The flagged corners (`mask`) of one cell by four lanes (gl = 0 .. 3, gmask).  Column n2 of a
// corner's matrix is read at the corner's vertex with its n2 bit cleared, so the values are
// s[(n2 N + n1) 4 + p] (3D: p the two other bits of the vertex) and s[n2 4 + n1 2 + p] (2D: p the
// other bit); lane gl loads and stores s[4 e + gl].
template <int DIM>
__device__ __forceinline__ void limit_cell(const LimiterArgs &a, int x, int y, int z, unsigned mask,
                                           int gl, unsigned gmask, double *s, const double *al,
                                           bool &capped) {
    constexpr int E = CellGrid<DIM>::kPerLane;
    const long V = (long)a.nx * a.ny * a.nz;
    double *src[DIM];  // of entry (n1, n2): src[n2] + n1 * DIM * V
    if constexpr (DIM == 3) {
        const int p = gl >> 1, q = gl & 1;
        src[0] = a.g + ((long)x * a.ny + (y + p)) * a.nz + (z + q);
        src[1] = a.g + V + ((long)(x + p) * a.ny + y) * a.nz + (z + q);
        src[2] = a.g + 2 * V + ((long)(x + p) * a.ny + (y + q)) * a.nz + z;
    } else {
        const int n1 = gl >> 1, p = gl & 1;
        src[0] = a.g + (n1 * 2) * V + (long)x * a.ny + (y + p);
        src[1] = a.g + (n1 * 2 + 1) * V + (long)(x + p) * a.ny + y;
    }
    double v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = DIM == 3 ? src[e / 3][(e % 3) * 3 * V] : *src[e % DIM];
#pragma unroll
    for (int e = 0; e < E; ++e) s[4 * e + gl] = v[e];
    __syncwarp(gmask);
    for (; mask; mask &= mask - 1) {
        const int c = __ffs((int)mask) - 1;
        // the corner's vertex: 000, 100, 010, 001, 011, 101, 110, 111, or 00, 10, 01, 11
        const int va = DIM == 3 ? 0xE2 >> c & 1 : c & 1, vb = DIM == 3 ? 0xD4 >> c & 1 : c >> 1,
                  vc = 0xB8 >> c & 1;
        const int col[3] = {DIM == 3 ? vb * 2 + vc : vb, DIM == 3 ? 12 + va * 2 + vc : 4 + va,
                            24 + va * 2 + vb};
        constexpr int kRow = DIM == 3 ? 4 : 2;
        double J[DIM][DIM];
#pragma unroll
        for (int n1 = 0; n1 < DIM; ++n1)
#pragma unroll
            for (int n2 = 0; n2 < DIM; ++n2) J[n1][n2] = s[col[n2] + n1 * kRow];
        // the entries this lane replaces: e = n2 DIM + n1 = gl, gl + 4, gl + 8
        constexpr int kOwn = DIM == 3 ? 3 : 1;
        double own[kOwn];
        int at[kOwn];
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            const int e = gl + 4 * i, n2 = e / DIM, n1 = e - n2 * DIM;
            at[i] = (n2 == 0 ? col[0] : n2 == 1 ? col[1] : col[2]) + n1 * kRow;
            own[i] = e < DIM * DIM ? s[at[i]] : 0.0;
        }
        // trial t: alpha after t steps; the lowest trial whose determinant is in range takes one
        // step more (trial 0 is J itself)
        int t = -1;
#pragma unroll 1
        for (int b = 0; b < kTrials && t < 0; b += 4) {
            const double at1 = al[b + gl];
            double Jn[DIM][DIM];
#pragma unroll
            for (int n1 = 0; n1 < DIM; ++n1)
#pragma unroll
                for (int n2 = 0; n2 < DIM; ++n2)
                    Jn[n1][n2] = (1 - at1) * J[n1][n2] + at1 * (n1 == n2 ? 1.0 : 0.0);
            const double det = detn<DIM>(Jn);
            const unsigned in = __ballot_sync(gmask, !(det > a.e2 || det < a.e1)) & gmask;
            if (in) t = b + ((__ffs((int)in) - 1) & 3);
        }
        if (t < 0) capped = true;
        const double alpha = al[t < 0 ? kTrials : t + 1];
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
            const int e = gl + 4 * i, n2 = e / DIM, n1 = e - n2 * DIM;
            if (e < DIM * DIM)
                s[at[i]] = (1 - alpha) * own[i] + alpha * (n1 == n2 ? 1.0 : 0.0);
        }
        __syncwarp(gmask);
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
        (DIM == 3 ? src[e / 3][(e % 3) * 3 * V] : *src[e % DIM]) = s[4 * e + gl];
    __syncwarp(gmask);  // the scratch is free for the group's next cell
}

// round 0: the flagged cells with no earlier flagged neighbour
__global__ void limiter_start_kernel(const LimiterArgs a) {
    const CellGrid<3> grid(a);
    const int cells = grid.count();
    for (int cell = blockIdx.x * blockDim.x + threadIdx.x; cell < cells;
         cell += gridDim.x * blockDim.x) {
        if (!a.mask[cell]) continue;
        const int n = grid.earlier_flagged(a.mask, cell);
        a.deg[cell] = n;
        if (n == 0) a.front[0][atomicAdd(&a.counts[0], 1)] = cell;
    }
}

// one round over the whole GPU
constexpr int kRoundThreads = 256;
__global__ void __launch_bounds__(kRoundThreads) limiter_round_kernel(const LimiterArgs a,
                                                                      int round) {
    __shared__ double al[kTrials + 1];
    __shared__ double scratch[kRoundThreads / 4 * CellGrid<3>::kStride];
    const int n = a.counts[round];
    if (blockIdx.x * (kRoundThreads / 4) >= n) return;
    if (threadIdx.x == 0) step_alphas(al);
    __syncthreads();
    const int gl = threadIdx.x & 3;
    const unsigned gmask = 0xfu << (threadIdx.x & 28);
    double *s = scratch + (threadIdx.x >> 2) * CellGrid<3>::kStride;
    const CellGrid<3> grid(a);
    const int *now = round & 1 ? a.front[1] : a.front[0];
    int *next = round & 1 ? a.front[0] : a.front[1];
    bool capped = false;
    for (int q = (blockIdx.x * kRoundThreads + threadIdx.x) >> 2; q < n;
         q += gridDim.x * (kRoundThreads / 4)) {
        const int cell = now[q];
        int x, y, z;
        grid.at(cell, x, y, z);
        limit_cell<3>(a, x, y, z, a.mask[cell], gl, gmask, s, al, capped);
        for (int l = gl; l < CellGrid<3>::kLater; l += 4) {
            const int nb = grid.neighbour(l, 1, x, y, z);
            if (nb >= 0 && a.mask[nb] && atomicSub(&a.deg[nb], 1) == 1)
                next[atomicAdd(&a.counts[round + 1], 1)] = nb;
        }
    }
    if (capped) atomicOr(a.flags, (unsigned)kFlagLimiterCapped);
}

// The rounds from `round` on, until none is left, in one CTA: small rounds cost less between two
// barriers than as launches.  SM: a grid of at most kSmallCells cells, all rounds, with the masks,
// counts and rounds in shared memory.  `groups` of four lanes have scratch.
constexpr int kSmallCells = 65536;
constexpr int kTailThreads = 1024;
template <int DIM, bool SM>
__global__ void __launch_bounds__(kTailThreads) limiter_tail_kernel(const LimiterArgs a, int round,
                                                                    int cap, int groups) {
    extern __shared__ __align__(16) unsigned char shm[];
    __shared__ int cnt[3];  // of this round, the next, and the one after (cleared meanwhile)
    __shared__ double al[kTrials + 1];
    const CellGrid<DIM> grid(a);
    const int cells = SM ? grid.count() : 0, words = (cells + 3) >> 2;
    double *scratch = reinterpret_cast<double *>(shm);  // [groups][kStride]
    unsigned *deg = reinterpret_cast<unsigned *>(scratch + (size_t)groups * grid.kStride);
    uint8_t *mask = reinterpret_cast<uint8_t *>(deg + words);                    // deg: 4 to a word
    unsigned short *f16 = reinterpret_cast<unsigned short *>(mask + 4 * words);  // [2][cap]
    const int tid = threadIdx.x, gl = tid & 3;
    const unsigned gmask = 0xfu << (tid & 28);
    if (tid < 3) cnt[tid] = 0;
    if (tid == 32) step_alphas(al);
    if (SM) {
        for (int i = tid; i < 4 * words; i += kTailThreads) mask[i] = i < cells ? a.mask[i] : 0;
        __syncthreads();
        for (int w = tid; w < words; w += kTailThreads) {
            unsigned d = 0;
            for (int e = 0; e < 4; ++e) {
                const int cell = 4 * w + e;
                if (cell >= cells || !mask[cell]) continue;
                const unsigned n = (unsigned)grid.earlier_flagged(mask, cell);
                d |= n << (8 * e);
                if (n == 0) f16[atomicAdd(&cnt[0], 1)] = (unsigned short)cell;
            }
            deg[w] = d;
        }
    } else {
        __syncthreads();
        if (tid == 0) cnt[0] = a.counts[round];
    }
    __syncthreads();
    bool capped = false;
    double *s = scratch + (size_t)(tid >> 2) * grid.kStride;
    for (int r = 0;; ++r, ++round) {
        const int n = cnt[r % 3], cur = round & 1;
        if (n == 0) break;  // uniform: nothing writes this count until the next barrier
        int *next = &cnt[(r + 1) % 3];
        if (tid < 4 * groups)
            for (int q = tid >> 2; q < n; q += groups) {
                const int cell = SM ? (int)f16[cur * cap + q]
                                    : (cur ? a.front[1] : a.front[0])[q];
                int x, y, z;
                grid.at(cell, x, y, z);
                limit_cell<DIM>(a, x, y, z, SM ? mask[cell] : a.mask[cell], gl, gmask, s, al,
                                capped);
                for (int l = gl; l < grid.kLater; l += 4) {
                    const int nb = grid.neighbour(l, 1, x, y, z);
                    if (nb < 0) continue;
                    if (SM) {
                        const int sh = 8 * (nb & 3);
                        if (mask[nb] && (atomicSub(&deg[nb >> 2], 1u << sh) >> sh & 0xffu) == 1u)
                            f16[(cur ^ 1) * cap + atomicAdd(next, 1)] = (unsigned short)nb;
                    } else if (a.mask[nb] && atomicSub(&a.deg[nb], 1) == 1) {
                        (cur ? a.front[0] : a.front[1])[atomicAdd(next, 1)] = nb;
                    }
                }
            }
        if (tid == 0) cnt[(r + 2) % 3] = 0;  // last read a barrier ago, next written a barrier on
        __syncthreads();                     // the round's gradients and the next round are complete
    }
    if (capped) atomicOr(a.flags, (unsigned)kFlagLimiterCapped);
}

// cells of a round at most: no two are neighbours
int most_apart(int cx, int cy, int cz) {
    return ((cx + 1) / 2) * ((cy + 1) / 2) * ((cz + 1) / 2);
}

constexpr int kMaxRounds = 24;  // rounds as launches of their own at most

// the limiter over every flagged cell; `corners`: how many corners are flagged
void launch_limiter(const LimiterArgs &a, long corners, cudaStream_t s) {
    const int cx = a.nx - 1, cy = a.ny - 1, cz = a.nz == 1 ? 1 : a.nz - 1;
    const long cells = (long)cx * cy * cz;
    if (cells <= kSmallCells) {
        const int cap = most_apart(cx, cy, cz);
        const size_t tables = (size_t)(cells + 3) / 4 * 8 + (size_t)cap * 4;
        auto launch = [&](auto dim) {
            constexpr int DIM = decltype(dim)::value;
            const size_t per = CellGrid<DIM>::kStride * sizeof(double), room = 226 * 1024 - tables;
            const int groups = room / per < kTailThreads / 4 ? (int)(room / per) : kTailThreads / 4;
            const size_t smem = groups * per + tables;
            BINDER_CUDA(cudaFuncSetAttribute(limiter_tail_kernel<DIM, true>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem));
            count_launch(), limiter_tail_kernel<DIM, true><<<1, kTailThreads, smem, s>>>(a, 0, cap,
                                                                                        groups);
        };
        if (a.nz == 1) launch(std::integral_constant<int, 2>());
        else launch(std::integral_constant<int, 3>());
        BINDER_CUDA(cudaGetLastError());
        return;
    }
    // the first rounds hold most of the cells of a field with many; a field with few is left to the
    // one CTA
    const int rounds = corners > 16384 ? kMaxRounds : (corners > 1024 ? 8 : 0);
    BINDER_CUDA(cudaMemsetAsync(a.counts, 0, sizeof(int) * (kMaxRounds + 1), s));
    long b = (cells + 255) / 256;
    const int grid = (int)(b < 148L * 16 ? b : 148L * 16);
    count_launch(), limiter_start_kernel<<<grid, 256, 0, s>>>(a);
    b = (corners + 63) / 64;
    const int rgrid = (int)(b < 148L * 8 ? b : 148L * 8);
    for (int r = 0; r < rounds; ++r)
        count_launch(), limiter_round_kernel<<<rgrid, kRoundThreads, 0, s>>>(a, r);
    constexpr int kGroups = kTailThreads / 4;
    const size_t smem = (size_t)kGroups * CellGrid<3>::kStride * sizeof(double);
    BINDER_CUDA(cudaFuncSetAttribute(limiter_tail_kernel<3, false>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    count_launch(), limiter_tail_kernel<3, false><<<1, kTailThreads, smem, s>>>(a, rounds, 0,
                                                                               kGroups);
    BINDER_CUDA(cudaGetLastError());
}

// backward-difference divergence (periodic) of each component's gradient row; the reference's
// Fourier factor (e^{-i theta} - 1) applied to the gradient spectra is minus its transform
__global__ void divergence_kernel(const double *g, int nx, int ny, int nz, double *div) {
    const long V = (long)nx * ny * nz;
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x) {
        const int x = (int)(p / ((long)ny * nz)), y = (int)((p / nz) % ny), z = (int)(p % nz);
        const int xm = x == 0 ? nx - 1 : x - 1, ym = y == 0 ? ny - 1 : y - 1,
                  zm = z == 0 ? nz - 1 : z - 1;
        const long px = ((long)xm * ny + y) * nz + z, py = ((long)x * ny + ym) * nz + z,
                   pz = ((long)x * ny + y) * nz + zm;
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const double *gx = g + (n * 3 + 0) * V, *gy = g + (n * 3 + 1) * V,
                         *gz = g + (n * 3 + 2) * V;
            div[n * V + p] = (gx[p] - gx[px]) + (gy[p] - gy[py]) + (gz[p] - gz[pz]);
        }
    }
}

// topology_correction_2D.cpp:165-207: the 4 corner Jacobians of every cell in the vertex order
// 00, 10, 01, 11 (the reference's Jff, Jbf, Jfb, Jbb), as a mask of those out of range.  Corner
// (vx, vy) pairs the x edge at y + vy with the y edge at x + vx (hi - lo each).  `below` / `above`
// count cells with a corner out of range, as the reference's counters do.  Positions are SoA [2][V].
__global__ void corner2d_kernel(const double *pos, int nx, int ny, double vol, double e1,
                                double e2, uint8_t *mask, Red *red) {
    const long V = (long)nx * ny;
    const long cy = ny - 1;
    const long cells = (long)(nx - 1) * cy;
    unsigned long long lb = 0, la = 0;
    for (long cell = (long)blockIdx.x * blockDim.x + threadIdx.x; cell < cells;
         cell += (long)gridDim.x * blockDim.x) {
        const int x = (int)(cell / cy), y = (int)(cell % cy);
        const long p00 = (long)x * ny + y, p10 = p00 + ny;
        const double X00 = pos[p00], X01 = pos[p00 + 1], X10 = pos[p10], X11 = pos[p10 + 1];
        const double Y00 = pos[V + p00], Y01 = pos[V + p00 + 1], Y10 = pos[V + p10],
                     Y11 = pos[V + p10 + 1];
        bool lo = false, hi = false;
        unsigned bits = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int vx = c & 1, vy = c >> 1;
            // x edge at y + vy, y edge at x + vx
            const double ex0 = vy ? X11 - X01 : X10 - X00, ex1 = vy ? Y11 - Y01 : Y10 - Y00;
            const double ey0 = vx ? X11 - X10 : X01 - X00, ey1 = vx ? Y11 - Y10 : Y01 - Y00;
            const double j = (ex0 * ey1 - ey0 * ex1) * vol;
            lo |= j < e1;
            hi |= j > e2;
            bits |= (j < e1 || j > e2) ? 1u << c : 0u;
        }
        mask[cell] = (uint8_t)bits;
        lb += lo;
        la += hi;
    }
    for (int o = 16; o > 0; o >>= 1) {
        lb += __shfl_xor_sync(0xffffffffu, lb, o);
        la += __shfl_xor_sync(0xffffffffu, la, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (lb) atomicAdd(&red->below, lb);
        if (la) atomicAdd(&red->above, la);
    }
}

// topology_correction_2D.cpp:209-246: periodic forward differences, g[(n1*2+n2)][p] =
// (pos_n1(p + e_n2) - pos_n1(p)) / vs[n1], and the sums of the positions into red
__global__ void gradient2d_kernel(const double *pos, int nx, int ny, double v0, double v1,
                                  double *g, Red *red) {
    const int V = nx * ny;
    double s[2] = {0.0, 0.0};
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < V; p += gridDim.x * blockDim.x) {
        const int x = p / ny, y = p - x * ny;
        const int px = x + 1 == nx ? y : p + ny;
        const int py = y + 1 == ny ? x * ny : p + 1;
        const double c0 = pos[p], c1 = pos[V + p];
        s[0] += c0;
        s[1] += c1;
        g[p] = (pos[px] - c0) / v0;
        g[V + p] = (pos[py] - c0) / v0;
        g[2 * V + p] = (pos[V + px] - c1) / v1;
        g[3 * V + p] = (pos[V + py] - c1) / v1;
    }
    add_sums(s, red);
}

// backward-difference divergence (periodic) of each component's 2D gradient row
__global__ void divergence2d_kernel(const double *g, int nx, int ny, double *div) {
    const long V = (long)nx * ny;
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x) {
        const int x = (int)(p / ny), y = (int)(p % ny);
        const long px = (long)(x == 0 ? nx - 1 : x - 1) * ny + y;
        const long py = (long)x * ny + (y == 0 ? ny - 1 : y - 1);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const double *gx = g + (n * 2 + 0) * V, *gy = g + (n * 2 + 1) * V;
            div[n * V + p] = (gx[p] - gx[px]) + (gy[p] - gy[py]);
        }
    }
}

// AoS grid-unit field [V][N] -> SoA physical [N][V] (times the voxel size) and back
struct Scale {
    double v[3];
};
__global__ void aos_to_soa_kernel(const double *aos, long V, int N, Scale sc, double *soa) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x)
        for (int n = 0; n < N; ++n) soa[n * V + p] = aos[p * N + n] * sc.v[n];
}
__global__ void soa_to_aos_kernel(const double *soa, long V, int N, Scale sc, double *aos) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x)
        for (int n = 0; n < N; ++n) aos[p * N + n] = soa[n * V + p] / sc.v[n];
}

int grid_for(long work) {
    int dev = 0, sms = 148;
    BINDER_CUDA(cudaGetDevice(&dev));
    BINDER_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long need = (work + 255) / 256;
    const long cap = (long)sms * 8;
    return (int)(need < 1 ? 1 : (need < cap ? need : cap));
}

// device buffer from the stream-ordered pool, released on the stream it was allocated on
template <typename T>
struct DBuf {
    T *p = nullptr;
    cudaStream_t s = 0;
    DBuf() = default;
    DBuf(size_t n, cudaStream_t stream) : s(stream) { p = dev_alloc_n<T>(n, s); }
    void alloc(size_t n, cudaStream_t stream) {
        dev_free(p, s);
        s = stream;
        p = dev_alloc_n<T>(n, s);
    }
    ~DBuf() { dev_free(p, s); }
    DBuf(const DBuf &) = delete;
    DBuf &operator=(const DBuf &) = delete;
};

void reset_red(Red *r, cudaStream_t s) {
    Red h{};
    h.mn = ~0ull;
    h.mx = 0ull;
    BINDER_CUDA(cudaMemcpyAsync(r, &h, sizeof(Red), cudaMemcpyHostToDevice, s));
}

Red read_red(const Red *r, cudaStream_t s) {
    Red h{};
    BINDER_CUDA(cudaMemcpyAsync(&h, r, sizeof(Red), cudaMemcpyDeviceToHost, s));
    BINDER_CUDA(cudaStreamSynchronize(s));
    return h;
}

}  // namespace

void jacobian3d_device(const double *field_aos, int nx, int ny, int nz, const double vs[3],
                       double *J, cudaStream_t s) {
    const long V = (long)nx * ny * nz;
    count_launch(), jacobian_kernel<<<grid_for(V), 256, 0, s>>>(field_aos, 3, 1, nx, ny, nz,
                                                1.0 / (vs[0] * vs[1] * vs[2]), J, 0.0, 0.0, nullptr);
    BINDER_CUDA(cudaGetLastError());
}

void jacobian2d_device(const double *field_aos, int nx, int ny, const double vs[2], double *J,
                       cudaStream_t s) {
    const long V = (long)nx * ny;
    count_launch(), jacobian2d_kernel<<<grid_for(V), 256, 0, s>>>(
                        field_aos, 2, 1, nx, ny, 1.0 / (vs[0] * vs[1]), J, 0.0, 0.0, nullptr);
    BINDER_CUDA(cudaGetLastError());
}

void jacobian2d(const double *field_host, int nx, int ny, const double vs[2], double *J_host) {
    BINDER_CHECK(nx > 0 && ny > 0, "dimensions must be positive");
    const long V = (long)nx * ny;
    cudaStream_t s = nullptr;
    BINDER_CUDA(cudaStreamCreate(&s));
    try {
        DBuf<double> f(V * 2, s), J(V, s);
        BINDER_CUDA(cudaMemcpyAsync(f.p, field_host, sizeof(double) * V * 2, cudaMemcpyHostToDevice, s));
        jacobian2d_device(f.p, nx, ny, vs, J.p, s);
        BINDER_CUDA(cudaMemcpyAsync(J_host, J.p, sizeof(double) * V, cudaMemcpyDeviceToHost, s));
        BINDER_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        cudaStreamSynchronize(s);
        cudaStreamDestroy(s);
        throw;
    }
    cudaStreamSynchronize(s);  // the buffers' stream-ordered frees
    cudaStreamDestroy(s);
}

// ---- Jacobian through a fixed device scratch array ------------------------------------------
// Some callers cannot afford cudaMalloc / cudaFree on every call: a framework whose caching
// allocator already holds most of the GPU's memory (a fresh cudaMalloc then fails even though the
// framework has room), or a loop that keeps other streams busy and cannot take the device-wide
// synchronisation cudaFree implies.  This variant stages the field, the determinants and the
// summary record in one array that is part of the library's device image, sized for grids of up
// to kJacobianNoAllocMaxVoxels voxels (16 MiB in all), so a call allocates nothing.
namespace {
constexpr size_t kNoAllocHeader = 256;  // the reduction record, padded
static_assert(sizeof(Red) <= kNoAllocHeader, "reduction record does not fit its slot");
// [Red | field: 3 * max doubles | J: max doubles]
static __device__ __align__(256) unsigned char
    g_jacobian_scratch[kNoAllocHeader + 4 * sizeof(double) * kJacobianNoAllocMaxVoxels];
constexpr int kNoAllocMaxDevices = 64;

// address of the scratch array on the current device, looked up once per device (with that
// device current) and kept for the life of the process; the lock guards only this table, not the
// scratch itself.  A cudaDeviceReset after the first call may place the module elsewhere in the
// next context, so the entry point does not support a device reset after its first call.
unsigned char *jacobian_scratch_address() {
    static std::mutex mu;
    static unsigned char *addr[kNoAllocMaxDevices] = {};
    int dev = -1;
    BINDER_CUDA(cudaGetDevice(&dev));
    BINDER_CHECK(dev >= 0 && dev < kNoAllocMaxDevices, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        BINDER_CUDA(cudaGetSymbolAddress(&p, g_jacobian_scratch));
        addr[dev] = static_cast<unsigned char *>(p);
    }
    return addr[dev];
}

// the record's starting values: min/max as empty ordered keys, counts zero
__global__ void clear_red_kernel(Red *r) {
    r->mn = ~0ull;
    r->mx = 0ull;
    r->below = r->above = r->negative = 0ull;
    r->sum[0] = r->sum[1] = r->sum[2] = 0.0;
    r->pad = 0;
}
}  // namespace

void jacobian3d_noalloc(const double *field_host, int nx, int ny, int nz, const double vs[3],
                        double *J_host, JacStats *stats) {
    BINDER_CHECK(nx > 0 && ny > 0 && nz > 0, "dimensions must be positive");
    const long V = (long)nx * ny * nz;
    if (V > kJacobianNoAllocMaxVoxels)
        throw Error(kInvalidArgument,
                    "grid of " + std::to_string(V) + " voxels exceeds the no-allocation limit of " +
                        std::to_string(kJacobianNoAllocMaxVoxels) + " voxels");
    unsigned char *base = jacobian_scratch_address();
    Red *red = reinterpret_cast<Red *>(base);
    double *df = reinterpret_cast<double *>(base + kNoAllocHeader);
    double *dj = df + 3 * kJacobianNoAllocMaxVoxels;
    // the calling thread's per-thread default stream: unlike the legacy stream 0 it does not
    // wait for (or hold up) work on the caller's other blocking streams
    const cudaStream_t s = cudaStreamPerThread;
    count_launch(), clear_red_kernel<<<1, 1, 0, s>>>(red);
    BINDER_CUDA(cudaGetLastError());
    BINDER_CUDA(cudaMemcpyAsync(df, field_host, sizeof(double) * V * 3, cudaMemcpyHostToDevice, s));
    // e1 = e2 = 0: `below` and `above` count J < 0 and J > 0
    count_launch(), jacobian_kernel<<<grid_for(V), 256, 0, s>>>(
        df, 3, 1, nx, ny, nz, 1.0 / (vs[0] * vs[1] * vs[2]), dj, 0.0, 0.0, red);
    BINDER_CUDA(cudaGetLastError());
    BINDER_CUDA(cudaMemcpyAsync(J_host, dj, sizeof(double) * V, cudaMemcpyDeviceToHost, s));
    Red h{};
    BINDER_CUDA(cudaMemcpyAsync(&h, red, sizeof(Red), cudaMemcpyDeviceToHost, s));
    BINDER_CUDA(cudaStreamSynchronize(s));
    if (stats) {
        stats->jmin = unordered(h.mn);
        stats->jmax = unordered(h.mx);
        stats->below = (long long)h.below;
        stats->above = (long long)h.above;
        stats->negative = (long long)h.negative;
    }
}

namespace {
__global__ void float_soa_to_physical_kernel(const float *d, long V, int N, Scale sc, double *pos) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x)
        for (int n = 0; n < N; ++n) pos[n * V + p] = (double)d[n * V + p] * sc.v[n];
}
__global__ void physical_to_float_soa_kernel(const double *pos, long V, int N, Scale sc, float *d) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < V;
         p += (long)gridDim.x * blockDim.x)
        for (int n = 0; n < N; ++n) d[n * V + p] = (float)(pos[n * V + p] / sc.v[n]);
}
}  // namespace

struct TopologyWorkspace::Impl {
    int nx, ny, nz;
    int N;  // 3, or 2 for an image (nz == 1)
    long V, cells;
    cudaStream_t st;  // pool stream of every buffer
    // always present: what the Jacobian statistics need
    DBuf<double> pos;
    DBuf<Red> red;
    DBuf<unsigned> flags;
    // allocated when a correction first iterates (most calls find every Jacobian in range)
    bool ready = false;
    DBuf<double> grad, div, t1, t2;
    DBuf<int> list, sorted;
    DBuf<uint8_t> mask;  // flagged corners per cell
    DBuf<int> deg, counts;
    HartleyMatrix H[3];
    DBuf<double> cs[3];
    Impl(int x, int y, int z, cudaStream_t s)
        : nx(x), ny(y), nz(z), N(z == 1 ? 2 : 3), V((long)x * y * z),
          cells(z == 1 ? (long)(x - 1) * (y - 1) : (long)(x - 1) * (y - 1) * (z - 1)), st(s),
          pos(V * N, s), red(1, s), flags(1, s) {}
    ~Impl() {
        for (auto &h : H) h.release(st);
    }
    void ensure() {
        if (ready) return;
        grad.alloc(V * N * N, st);
        mask.alloc(cells, st);
        if (cells > kSmallCells) {  // the limiter's rounds in global memory
            deg.alloc(cells, st);
            counts.alloc(kMaxRounds + 1, st);
            list.alloc(cells, st);
            sorted.alloc(cells, st);
        }
        div.alloc(V * N, st);
        t1.alloc(V * N, st);
        t2.alloc(V * N, st);
        const int dims[3] = {nx, ny, nz};
        const double pi = 3.14159265358979323846;
        for (int a = 0; a < 3; ++a) {
            const int n = dims[a];
            H[a].init(n, st);
            cs[a].alloc(n, st);
            std::vector<double> c(n);
            for (int k = 0; k < n; ++k) c[k] = std::cos(2.0 * pi * k / (n * 1.0));
            BINDER_CUDA(cudaMemcpyAsync(cs[a].p, c.data(), sizeof(double) * n,
                                        cudaMemcpyHostToDevice, st));
            BINDER_CUDA(cudaStreamSynchronize(st));  // `c` goes out of scope
        }
        ready = true;
    }
};

TopologyWorkspace::TopologyWorkspace(int nx, int ny, int nz, cudaStream_t s) {
    BINDER_CHECK(nx >= 2 && ny >= 2 && (nz >= 2 || nz == 1),
                 "topology correction needs at least 2 voxels per axis (nz == 1 for an image)");
    BINDER_CHECK(nx <= 256 && ny <= 256 && nz <= 256, "topology correction supports axes up to 256");
    impl_ = new Impl(nx, ny, nz, s);
}
TopologyWorkspace::~TopologyWorkspace() { delete impl_; }
double *TopologyWorkspace::positions() { return impl_->pos.p; }

// BINDER/src/cpu/topology_correction_3D.cpp:17-143 on the workspace's SoA physical positions
TopologyResult TopologyWorkspace::run(double e1, double e2, int max_outer, int max_inner,
                                      const double vs[3], cudaStream_t s) {
    if (impl_->N == 2) return run2d(e1, e2, max_outer, max_inner, vs, s);
    BINDER_CHECK(vs[0] > 0 && vs[1] > 0 && vs[2] > 0, "voxel sizes must be positive");
    Impl &w = *impl_;
    const int nx = w.nx, ny = w.ny, nz = w.nz;
    const long V = w.V, cells = w.cells;
    const double vol = 1.0 / (vs[0] * vs[1] * vs[2]);
    // powers of two, with reciprocals that are too
    bool exact = true;
    for (int n = 0; n < 3; ++n) {
        int e = 0;
        exact = exact && std::frexp(vs[n], &e) == 0.5 && std::isfinite(1.0 / vs[n]);
    }
    TopologyResult res{};
    BINDER_CUDA(cudaMemsetAsync(w.flags.p, 0, sizeof(unsigned), s));

    auto jac_stats = [&]() {
        reset_red(w.red.p, s);
        count_launch(), jacobian_kernel<<<grid_for(V), 256, 0, s>>>(w.pos.p, 1, V, nx, ny, nz, vol, nullptr, e1, e2,
                                                    w.red.p);
        BINDER_CUDA(cudaGetLastError());
        return read_red(w.red.p, s);
    };
    auto corners = [&]() {
        reset_red(w.red.p, s);
        count_launch(), corner_kernel<<<grid_for(cells), 256, 0, s>>>(w.pos.p, nx, ny, nz, vol, e1, e2,
                                                                      w.mask.p, w.red.p);
        BINDER_CUDA(cudaGetLastError());
        return read_red(w.red.p, s);
    };

    Red r = jac_stats();
    double jmin = unordered(r.mn), jmax = unordered(r.mx);
    res.below_before = (long long)r.below;
    res.above_before = (long long)r.above;
    int outer = 0;
    while ((jmin < e1 || jmax > e2) && outer < max_outer) {
        w.ensure();
        Red c = corners();
        int inner = 0;
        while ((c.below > 0 || c.above > 0) && inner < max_inner) {
            // (the sums of the positions onto the zeros that corners() left)
            count_launch();
            if (exact)
                gradient_kernel<true><<<grid_for(V), 256, 0, s>>>(
                    w.pos.p, nx, ny, nz, 1.0 / vs[0], 1.0 / vs[1], 1.0 / vs[2], w.grad.p, w.red.p);
            else
                gradient_kernel<false><<<grid_for(V), 256, 0, s>>>(
                    w.pos.p, nx, ny, nz, vs[0], vs[1], vs[2], w.grad.p, w.red.p);
            LimiterArgs la{};
            la.mask = w.mask.p;
            la.g = w.grad.p;
            la.deg = w.deg.p;
            la.front[0] = w.list.p;
            la.front[1] = w.sorted.p;
            la.counts = w.counts.p;
            la.nx = nx; la.ny = ny; la.nz = nz;
            la.e1 = e1; la.e2 = e2;
            la.flags = w.flags.p;
            launch_limiter(la, (long)(c.below + c.above), s);
            BINDER_CUDA(cudaGetLastError());
            count_launch(), divergence_kernel<<<grid_for(V), 256, 0, s>>>(w.grad.p, nx, ny, nz, w.div.p);
            BINDER_CUDA(cudaGetLastError());

            // u = -(1/V) H (H div / lambda): separable Hartley passes z, y, [x fused], y, z
            HartleyArgs a{};
            a.V = V;
            a.nz = nz;
            a.cos_x = w.cs[0].p;
            a.cos_y = w.cs[1].p;
            a.cos_z = w.cs[2].p;
            a.in = w.div.p; a.out = w.t1.p; a.outer = (long)nx * ny; a.s = 1;
            launch_hartley(a, w.H[2], kHartleyPlain, 3, s);
            a.in = w.t1.p; a.out = w.t2.p; a.outer = nx; a.s = nz;
            launch_hartley(a, w.H[1], kHartleyPlain, 3, s);
            a.in = w.t2.p; a.out = w.t1.p; a.outer = 1; a.s = (long)ny * nz;
            launch_hartley(a, w.H[0], kHartleyPoisson, 3, s);
            a.in = w.t1.p; a.out = w.t2.p; a.outer = nx; a.s = nz;
            launch_hartley(a, w.H[1], kHartleyPlain, 3, s);
            // last pass: physical positions u * vs + mean
            a.in = w.t2.p; a.out = w.pos.p; a.outer = (long)nx * ny; a.s = 1;
            for (int n = 0; n < 3; ++n) a.out_scale[n] = vs[n];
            a.sums = w.red.p->sum;
            a.count = nx * ny * nz;
            launch_hartley(a, w.H[2], kHartleyScaled, 3, s);
            c = corners();
            inner++;
            res.inner_iterations++;
        }
        r = jac_stats();
        jmin = unordered(r.mn);
        jmax = unordered(r.mx);
        outer++;
    }
    res.outer_iterations = outer;
    res.below_after = (long long)r.below;
    res.above_after = (long long)r.above;
    BINDER_CUDA(cudaMemcpyAsync(&res.flags, w.flags.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    BINDER_CUDA(cudaStreamSynchronize(s));
    return res;
}

// BINDER/src/cpu/topology_correction_2D.cpp:17-163: the 3D loop structure with 4 corners per
// cell, 2x2 gradient matrices and a 2D Poisson solve (separable Hartley passes y, [x fused], y)
TopologyResult TopologyWorkspace::run2d(double e1, double e2, int max_outer, int max_inner,
                                        const double vs[3], cudaStream_t s) {
    BINDER_CHECK(vs[0] > 0 && vs[1] > 0, "voxel sizes must be positive");
    Impl &w = *impl_;
    const int nx = w.nx, ny = w.ny;
    const long V = w.V, cells = w.cells;
    const double vol = 1.0 / (vs[0] * vs[1]);
    TopologyResult res{};
    BINDER_CUDA(cudaMemsetAsync(w.flags.p, 0, sizeof(unsigned), s));

    auto jac_stats = [&]() {
        reset_red(w.red.p, s);
        count_launch(), jacobian2d_kernel<<<grid_for(V), 256, 0, s>>>(w.pos.p, 1, V, nx, ny, vol,
                                                                      nullptr, e1, e2, w.red.p);
        BINDER_CUDA(cudaGetLastError());
        return read_red(w.red.p, s);
    };
    auto corners = [&]() {
        reset_red(w.red.p, s);
        count_launch(), corner2d_kernel<<<grid_for(cells), 256, 0, s>>>(w.pos.p, nx, ny, vol, e1,
                                                                        e2, w.mask.p, w.red.p);
        BINDER_CUDA(cudaGetLastError());
        return read_red(w.red.p, s);
    };

    Red r = jac_stats();
    double jmin = unordered(r.mn), jmax = unordered(r.mx);
    res.below_before = (long long)r.below;
    res.above_before = (long long)r.above;
    int outer = 0;
    while ((jmin < e1 || jmax > e2) && outer < max_outer) {
        w.ensure();
        Red c = corners();
        int inner = 0;
        while ((c.below > 0 || c.above > 0) && inner < max_inner) {
            // (the sums of the positions onto the zeros that corners() left)
            count_launch(), gradient2d_kernel<<<grid_for(V), 256, 0, s>>>(w.pos.p, nx, ny, vs[0],
                                                                          vs[1], w.grad.p, w.red.p);
            LimiterArgs la{};
            la.mask = w.mask.p;
            la.g = w.grad.p;
            la.nx = nx; la.ny = ny; la.nz = 1;
            la.e1 = e1; la.e2 = e2;
            la.flags = w.flags.p;
            launch_limiter(la, (long)(c.below + c.above), s);
            BINDER_CUDA(cudaGetLastError());
            count_launch(), divergence2d_kernel<<<grid_for(V), 256, 0, s>>>(w.grad.p, nx, ny,
                                                                            w.div.p);
            BINDER_CUDA(cudaGetLastError());

            // u = -(1/V) H (H div / lambda) on the nx x ny grid (the volume nx x ny x 1, whose
            // unit z axis contributes cos 0 = 1 to lambda = 6 - 2cos_x - 2cos_y - 2cos_z)
            HartleyArgs a{};
            a.V = V;
            a.nz = 1;
            a.cos_x = w.cs[0].p;
            a.cos_y = w.cs[1].p;
            a.cos_z = w.cs[2].p;
            a.in = w.div.p; a.out = w.t1.p; a.outer = nx; a.s = 1;
            launch_hartley(a, w.H[1], kHartleyPlain, 2, s);
            a.in = w.t1.p; a.out = w.t2.p; a.outer = 1; a.s = ny;
            launch_hartley(a, w.H[0], kHartleyPoisson, 2, s);
            // last pass: physical positions u * vs + mean
            a.in = w.t2.p; a.out = w.pos.p; a.outer = nx; a.s = 1;
            for (int n = 0; n < 2; ++n) a.out_scale[n] = vs[n];
            a.sums = w.red.p->sum;
            a.count = nx * ny;
            launch_hartley(a, w.H[1], kHartleyScaled, 2, s);
            c = corners();
            inner++;
            res.inner_iterations++;
        }
        r = jac_stats();
        jmin = unordered(r.mn);
        jmax = unordered(r.mx);
        outer++;
    }
    res.outer_iterations = outer;
    res.below_after = (long long)r.below;
    res.above_after = (long long)r.above;
    BINDER_CUDA(cudaMemcpyAsync(&res.flags, w.flags.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    BINDER_CUDA(cudaStreamSynchronize(s));
    return res;
}

void TopologyWorkspace::load_float_grid(const float *d_soa, const double vs[3], cudaStream_t s) {
    const Scale sc{{vs[0], vs[1], vs[2]}};
    count_launch(), float_soa_to_physical_kernel<<<grid_for(impl_->V), 256, 0, s>>>(
                        d_soa, impl_->V, impl_->N, sc, impl_->pos.p);
    BINDER_CUDA(cudaGetLastError());
}

void TopologyWorkspace::store_float_grid(float *d_soa, const double vs[3], cudaStream_t s) {
    const Scale sc{{vs[0], vs[1], vs[2]}};
    count_launch(), physical_to_float_soa_kernel<<<grid_for(impl_->V), 256, 0, s>>>(
                        impl_->pos.p, impl_->V, impl_->N, sc, d_soa);
    BINDER_CUDA(cudaGetLastError());
}

TopologyResult topology_correct_3d(double *host, double e1, double e2, int max_outer,
                                   int max_inner, const double vs[3], int nx, int ny, int nz,
                                   cudaStream_t s) {
    BINDER_CHECK(vs[0] > 0 && vs[1] > 0 && vs[2] > 0, "voxel sizes must be positive");
    BINDER_CHECK(nz >= 2, "a 3D field needs nz >= 2 (use the 2D entry point for images)");
    return topology_correct(host, e1, e2, max_outer, max_inner, vs, nx, ny, nz, s);
}

TopologyResult topology_correct_2d(double *host, double e1, double e2, int max_outer,
                                   int max_inner, const double vs[2], int nx, int ny,
                                   cudaStream_t s) {
    BINDER_CHECK(vs[0] > 0 && vs[1] > 0, "voxel sizes must be positive");
    const double vs3[3] = {vs[0], vs[1], 1.0};
    return topology_correct(host, e1, e2, max_outer, max_inner, vs3, nx, ny, 1, s);
}

// host AoS field (grid units) -> device SoA physical -> correction -> back, in place
TopologyResult topology_correct(double *host, double e1, double e2, int max_outer, int max_inner,
                                const double vs[3], int nx, int ny, int nz, cudaStream_t s) {
    TopologyWorkspace ws(nx, ny, nz, s);
    const long V = (long)nx * ny * nz;
    const int N = nz == 1 ? 2 : 3;
    const Scale sc{{vs[0], vs[1], vs[2]}};
    DBuf<double> aos(V * N, s);
    BINDER_CUDA(cudaMemcpyAsync(aos.p, host, sizeof(double) * V * N, cudaMemcpyHostToDevice, s));
    count_launch(), aos_to_soa_kernel<<<grid_for(V), 256, 0, s>>>(aos.p, V, N, sc, ws.positions());
    BINDER_CUDA(cudaGetLastError());
    TopologyResult res = ws.run(e1, e2, max_outer, max_inner, vs, s);
    count_launch(), soa_to_aos_kernel<<<grid_for(V), 256, 0, s>>>(ws.positions(), V, N, sc, aos.p);
    BINDER_CUDA(cudaGetLastError());
    BINDER_CUDA(cudaMemcpyAsync(host, aos.p, sizeof(double) * V * N, cudaMemcpyDeviceToHost, s));
    BINDER_CUDA(cudaStreamSynchronize(s));
    return res;
}

}  // namespace binder
