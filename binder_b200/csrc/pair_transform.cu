// Two DCT passes per launch (tcgen05 / TMEM): the M-step of a volume in three launches instead of
// six, with half the field traffic.
//
// The M-step transforms every line along z, y, x, scales, and transforms back along x, y, z
// (BINDER/src/cpu/NonLinearTransformation.cpp:58-126).  Each pair of neighbouring passes works on
// independent pieces that fit on one SM, so a CTA keeps the field between the two passes in shared
// memory:
//   kPairForward   one (y, z) plane and a tile of its kz: D1[kz][y] = sum_z Cz[kz][z] X[y][z], then
//                  D2[kz][ky] = sum_y D1[kz][y] Cy[ky][y].  A plane with more than 128 kz is
//                  shared by several CTAs, each reading the plane and storing its kz.
//   kPairSpectral  128 neighbouring (ky, kz) lines: D1[t][kx], the prior scaling (noise, costs),
//                  D2[t][x].  Reads and writes the same lines, so it runs in place.
//   kPairInverse   one (ky, kz) plane and a tile of its y: D1[y][kz] = sum_ky Cy[ky][y] X[ky][kz],
//                  then D2[z][y] = sum_kz Cz[kz][z] D1[y][kz], voxel positions added.
// The operand roles (data as A or as B) are chosen so that both operands are K-major, the
// intermediate goes from TMEM to shared memory in 16-byte stores, and the lanes of the last
// accumulator run along the contiguous axis, so stores are coalesced without staging.
//
// A persistent CTA per SM (two where tiles are small) walks the tiles.  Warps: load warps, epilogue
// warps, one MMA warp, one matrix-copy warp.  Load warps keep two steps of 32 K in flight in
// registers, split them into BF16 hi / lo and store them into a ring; the matrices come by
// cp.async.bulk into a ring of their own; the epilogue warps move the first accumulator into the
// second product's operand and the second accumulator to global memory while the MMA warp and the
// load warps are on the next tile.
//
// What bounds it (160x192x160, per tile of 8 us): the single issuing thread of the MMAs (7.2 us)
// and the epilogue warps (7.5 us), neither HBM (a pass moves 118 MB, 18 us of its 65 us) nor the
// matrix copies (without them 2% less).  Measured against the six per-axis passes on three streams:
// M-step 0.294 -> 0.195 ms at 160x192x160, 58 -> 38 us at 96^3, 51 -> 27 us at 64^3; the passes of
// a sweep of 32 chains at 96^3 1.67 -> 0.82 ms.
// Tried on the way: one CTA per tile with the same warps loading and storing 0.296 ms; the steps of
// the MMA warp one K chunk of 16 long 0.264 ms (its waits and commits took as long as its MMAs);
// one group of load warps instead of two 0.240 ms; 32 accumulator columns per TMEM load instead of
// 16 0.233 ms (spills); waits that poll instead of suspending 0.202 ms.
// Bit for bit the per-axis passes: the same K chunks of 16 in the same order, the same three
// products (data hi x matrix hi, data hi x matrix lo, data lo x matrix hi), FP32 between passes.
#include <algorithm>

#include "layout.cuh"
#include "pair_transform.cuh"
#include "transform.cuh"
#include "umma.cuh"
#include <cuda_bf16.h>

namespace binder {
namespace {

constexpr uint64_t kPairWait = 2000000000ull;  // 2 s of wall time per barrier wait
constexpr int kMaxAxis = 256;                  // MMA N, and 16 K chunks
constexpr int kMaxSteps = kMaxAxis / 32;       // pipeline steps of 32 K (two MMA chunks of 16)
constexpr int kMaxRing = 16;  // operand ring slots at most
constexpr int kMaxMat = 6;    // matrix ring slots at most
constexpr int kSlack = 2048;  // an A operand of fewer than 128 rows is read past its end

struct PairArgs {
    const float *in;
    float *out;
    long V;
    const unsigned char *m1, *m2;  // BF16 chunks [nk][2 planes][2 K columns][np rows][16 bytes]
    int np1, np2;                  // rows of the matrices (padded to 16)
    int nk1, nk2;                  // K chunks (of 16) of the two products
    int nx, ny, nz;
    long lines;       // kPairSpectral: lines (= line stride along x)
    int rp;           // rows of the loaded operand in shared memory
    int tm, tiles;    // rows of the tiled output axis per tile, tiles per plane
    long ctas;        // tiles per component
    long total;       // tiles of the launch
    int mats;         // matrix ring slots
    int ring;         // operand ring slots
    uint32_t ring_off, mat_off, mat_slot, bar_off;  // bytes
    uint32_t ncols;   // TMEM columns
    const float *D;
    DevState *st;
    double sigma2;
    int sample, want_raw, every;
    const float *noise;
    double rho_p;
    double eta2[3];
    const float *xpos;
    int dims;
    int comp0, chain_comps;
    int ring_n;
    long ring_stride;
    const int *skip;
};

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(dst), "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(umma::smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

// eight FP32 values as BF16 hi (round to nearest even) and, with PLANES == 2, lo = BF16(x - hi):
// one 16-byte row of a K column per plane, the planes `plane` bytes apart
template <int PLANES>
__device__ __forceinline__ void split8(unsigned char *dst, uint32_t plane, const float *v) {
    uint32_t h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        h[i] = *reinterpret_cast<const uint32_t *>(&b);
    }
    *reinterpret_cast<uint4 *>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    if (PLANES == 2) {
        uint32_t l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 d = __fadd2_rn(make_float2(v[2 * i], v[2 * i + 1]),
                                        make_float2(-__uint_as_float(h[i] << 16),
                                                    -__uint_as_float(h[i] & 0xffff0000u)));
            const __nv_bfloat162 b = __float22bfloat162_rn(d);
            l[i] = *reinterpret_cast<const uint32_t *>(&b);
        }
        *reinterpret_cast<uint4 *>(dst + plane) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// one K chunk of 16: A rows `pa` and B rows `pb` apart in their K columns, planes 32 rows' bytes
// apart; DATA_A: the data (not the matrix) is operand A
template <int PLANES, bool DATA_A>
__device__ __forceinline__ void mma_chunk(uint32_t d, uint32_t a, uint32_t pa, uint32_t b,
                                          uint32_t pb, uint32_t idesc, bool first) {
    const uint64_t ahi = umma::smem_desc(a, pa * 16u, 128u);
    const uint64_t bhi = umma::smem_desc(b, pb * 16u, 128u);
    umma::mma_bf16(d, ahi, bhi, idesc, first ? 0u : 1u);
    if (PLANES == 2) {
        const uint64_t alo = umma::smem_desc(a + pa * 32u, pa * 16u, 128u);
        const uint64_t blo = umma::smem_desc(b + pb * 32u, pb * 16u, 128u);
        umma::mma_bf16(d, DATA_A ? ahi : alo, DATA_A ? blo : bhi, idesc, 1u);
        umma::mma_bf16(d, DATA_A ? alo : ahi, DATA_A ? bhi : blo, idesc, 1u);
    }
}

// the output tile a CTA works on: component, plane and tile of the plane
struct Tile {
    int comp, plane, row0;  // row0: first kz / y / line
    long base;              // element of `in` / `out` the plane (the tile of lines) starts at
};

template <int KIND>
__device__ __forceinline__ Tile tile_at(const PairArgs &a, int i) {
    const unsigned t = blockIdx.x + (unsigned)i * gridDim.x;
    Tile r;
    r.comp = (int)(t / (unsigned)a.ctas);
    const unsigned rem = t - (unsigned)r.comp * (unsigned)a.ctas;
    r.plane = KIND == kPairSpectral ? 0 : (int)(rem / (unsigned)a.tiles);
    const int tile = (int)rem - r.plane * (KIND == kPairSpectral ? 0 : a.tiles);
    r.row0 = tile * (KIND == kPairSpectral ? 128 : a.tm);
    r.comp += a.comp0;
    r.base = (long)r.comp * a.V +
             (KIND == kPairSpectral ? (long)r.row0 : (long)r.plane * a.ny * a.nz);
    return r;
}

// NL load warps, NE epilogue warps, one MMA warp and one matrix-copy warp
// VAR: kPairForward: rows of whole float4 (nz % 4 == 0); kPairSpectral: with the prior noise
template <int KIND, int PLANES, int NL, int NE, bool VAR>
__global__ void __launch_bounds__((NL + NE + 2) * 32, NE == 4 ? 2 : 1) pair_kernel(const PairArgs a) {
    constexpr int kMma = NL + NE;  // the MMA warp
    // eight load warps or more work in two groups on alternate steps: two steps in flight
    constexpr int kGroups = NL >= 8 ? 2 : 1;
    constexpr int GW = NL / kGroups;  // warps per group
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint64_t *xfull = reinterpret_cast<uint64_t *>(smem + a.bar_off);  // [kMaxRing]
    uint64_t *xfree = xfull + kMaxRing;                                // [kMaxRing]
    uint64_t *dready = xfree + kMaxRing;                               // [kMaxSteps]
    uint64_t *mfull = dready + kMaxSteps;                              // [kMaxMat]
    uint64_t *mfree = mfull + kMaxMat;                                 // [kMaxMat]
    uint64_t *d1full = mfree + kMaxMat, *d2full = d1full + 1, *d2free = d1full + 2,
             *drain = d1full + 3;
    uint32_t *holder = reinterpret_cast<uint32_t *>(drain + 1);
    int *s_err = reinterpret_cast<int *>(holder + 1);
    volatile int *err = s_err;

    // rows of the loaded operand and of the intermediate's K columns
    const uint32_t rp = KIND == kPairSpectral ? 128u : (uint32_t)a.rp;
    const uint32_t tm = KIND == kPairSpectral ? 128u : (uint32_t)a.tm;
    const uint32_t xchunk = (uint32_t)PLANES * 32u * rp;  // bytes of one K chunk of 16
    const uint32_t dchunk = (uint32_t)PLANES * 32u * tm;
    const int ns1 = (a.nk1 + 1) >> 1, ns2 = (a.nk2 + 1) >> 1;  // steps of the two products
    // tiles of this CTA: blockIdx.x, blockIdx.x + gridDim.x, ...
    const int mine = (int)((a.total - blockIdx.x + gridDim.x - 1) / gridDim.x);

    if (warp == NL) umma::tmem_alloc(holder, a.ncols);
    if (tid == 0) {
        for (int i = 0; i < kMaxRing; ++i) {
            umma::mbar_init(&xfull[i], GW);
            umma::mbar_init(&xfree[i], 1);
        }
        for (int i = 0; i < kMaxSteps; ++i) umma::mbar_init(&dready[i], 4);
        for (int i = 0; i < kMaxMat; ++i) {
            umma::mbar_init(&mfull[i], 1);
            umma::mbar_init(&mfree[i], 1);
        }
        umma::mbar_init(d1full, 1);
        umma::mbar_init(d2full, 1);
        umma::mbar_init(d2free, NE);
        umma::mbar_init(drain, 1);
        *s_err = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *holder;
    const uint32_t sbase = umma::smem_u32(smem);
    // 32-bit offsets from the plane's (or the tile's) first element: V < 2^31
    const uint32_t ks = KIND == kPairSpectral ? (uint32_t)a.lines : (uint32_t)a.nz;

    if (warp == kMma) {
        // ---- MMA warp: one lane.  A chunk's three MMAs issue in 0.18 us; the waits, fences and
        // commits around them took as long again with one chunk of 16 per step, so a step is two
        if (lane == 0) {
            const uint32_t n1 = KIND == kPairSpectral ? (uint32_t)a.np1 : rp;
            const uint32_t n2 = KIND == kPairInverse ? tm : (uint32_t)a.np2;
            const uint32_t id1 = umma::instr_desc(128, (int)n1, umma::kFmtBF16);
            const uint32_t id2 = umma::instr_desc(128, (int)n2, umma::kFmtBF16);
            const uint32_t mrows = KIND == kPairSpectral ? (uint32_t)a.np1 : tm;
            const uint32_t mchunk1 = (uint32_t)PLANES * 32u * mrows;
            const uint32_t mchunk2 = (uint32_t)PLANES * 32u * (uint32_t)a.np2;
            const uint32_t d2 = tmem + n1;  // columns of the second accumulator
            bool ok = true;
            int ms = 0, xs = 0;
            uint32_t mph = 0, xph = 0;
            for (int i = 0; i < mine && ok; ++i) {
                for (int s = 0; s < ns1; ++s) {
                    ok = umma::mbar_wait(&xfull[xs], xph, kPairWait) &&
                         umma::mbar_wait(&mfull[ms], mph, kPairWait);
                    if (!ok) break;
                    umma::fence_after_sync();
                    const uint32_t x = sbase + a.ring_off + (uint32_t)xs * 2u * xchunk;
                    const uint32_t m = sbase + a.mat_off + (uint32_t)ms * a.mat_slot;
                    for (int q = 0; q < 2 && 2 * s + q < a.nk1; ++q) {
                        const uint32_t xq = x + (uint32_t)q * xchunk;
                        const uint32_t mq = m + (uint32_t)q * mchunk1;
                        if (KIND == kPairSpectral)
                            mma_chunk<PLANES, true>(tmem, xq, rp, mq, mrows, id1, s + q == 0);
                        else
                            mma_chunk<PLANES, false>(tmem, mq, mrows, xq, rp, id1, s + q == 0);
                    }
                    umma::commit(&xfree[xs]);
                    umma::commit(&mfree[ms]);
                    if (++xs == a.ring) xs = 0, xph ^= 1;
                    if (++ms == a.mats) ms = 0, mph ^= 1;
                }
                if (!ok) break;
                umma::commit(d1full);
                // the second accumulator was read by every epilogue warp
                if (i > 0) ok = umma::mbar_wait(d2free, (uint32_t)(i - 1) & 1u, kPairWait);
                for (int s = 0; s < ns2 && ok; ++s) {
                    ok = umma::mbar_wait(&dready[s], (uint32_t)i & 1u, kPairWait) &&
                         umma::mbar_wait(&mfull[ms], mph, kPairWait);
                    if (!ok) break;
                    umma::fence_after_sync();
                    const uint32_t x = sbase + (uint32_t)s * 2u * dchunk;
                    const uint32_t m = sbase + a.mat_off + (uint32_t)ms * a.mat_slot;
                    for (int q = 0; q < 2 && 2 * s + q < a.nk2; ++q) {
                        const uint32_t xq = x + (uint32_t)q * dchunk;
                        const uint32_t mq = m + (uint32_t)q * mchunk2;
                        if (KIND == kPairInverse) {
                            for (int t = 0; t * 128 < a.np2; ++t)
                                mma_chunk<PLANES, false>(d2 + (uint32_t)t * tm,
                                                         mq + (uint32_t)t * 2048u, (uint32_t)a.np2,
                                                         xq, tm, id2, s + q == 0);
                        } else {
                            mma_chunk<PLANES, true>(d2, xq, tm, mq, (uint32_t)a.np2, id2,
                                                    s + q == 0);
                        }
                    }
                    umma::commit(&mfree[ms]);
                    if (++ms == a.mats) ms = 0, mph ^= 1;
                }
                if (ok) umma::commit(d2full);
            }
            if (!ok) *err = 1;
        }
    } else if (warp == kMma + 1) {
        // ---- matrix copies: the steps of both products, a.mats ahead -----------------------------
        if (lane == 0) {
            int issued = 0, slot = 0;
            uint32_t ph = 1;  // phase of mfree: the first round finds every slot free
            bool ok = true;
            for (int i = 0; i < mine && ok; ++i) {
                const int row0 = tile_at<KIND>(a, i).row0;
                // this tile's rows of every K column (the last tile may have fewer)
                const uint32_t rows = min(tm, (uint32_t)(a.np1 - row0));
                for (int c = 0; c < ns1 + ns2; ++c) {
                    if (issued >= a.mats && (!umma::mbar_wait(&mfree[slot], ph, kPairWait) || *err)) {
                        ok = false;
                        break;
                    }
                    const uint32_t dst = sbase + a.mat_off + (uint32_t)slot * a.mat_slot;
                    const uint32_t bar = umma::smem_u32(&mfull[slot]);
                    const bool second = c >= ns1;
                    const int k0 = 2 * (second ? c - ns1 : c);  // first chunk of the step
                    const uint32_t nq = (uint32_t)min(2, (second ? a.nk2 : a.nk1) - k0);
                    const uint32_t np = second ? a.np2 : a.np1;
                    const unsigned char *src = (second ? a.m2 : a.m1) + (size_t)k0 * 64u * np;
                    if (!second && KIND != kPairSpectral) {
                        expect_tx(&mfull[slot], nq * PLANES * 2u * rows * 16u);
                        for (uint32_t q = 0; q < nq; ++q)
#pragma unroll
                            for (uint32_t e = 0; e < 2 * PLANES; ++e)
                                bulk_copy(dst + (q * 2u * PLANES + e) * tm * 16u,
                                          src + (size_t)(q * 4u + e) * np * 16u + row0 * 16,
                                          rows * 16u, bar);
                    } else {
                        expect_tx(&mfull[slot], nq * PLANES * 32u * np);
                        if (PLANES == 2) {
                            bulk_copy(dst, src, nq * 64u * np, bar);
                        } else {
                            for (uint32_t q = 0; q < nq; ++q)
                                bulk_copy(dst + q * 32u * np, src + (size_t)q * 64u * np, 32u * np,
                                          bar);
                        }
                    }
                    ++issued;
                    if (++slot == a.mats) slot = 0, ph ^= 1;
                }
            }
            if (!ok) *err = 1;
            // after an error nothing waits for the last copies: let them land before the exit
            if (*err)
                for (int g = max(0, issued - a.mats); g < issued; ++g)
                    umma::mbar_wait(&mfull[g % a.mats], (uint32_t)(g / a.mats) & 1u, kPairWait);
        }
    } else if (warp < NL) {
        // ---- load warps ------------------------------------------------------------------------
        // One step of 32 K: a warp's tasks are 8 rows x 32 K (contiguous rows, 128 bytes each) or
        // 32 rows x 8 K (strided), at most four; they are split and stored, published with one
        // fence and one arrival, and the next step's are loaded (the next tile is on its way to L2
        // by then).
        constexpr bool kContig = KIND == kPairForward;
        constexpr int kTasks = 4;  // GW * 32 rows at most: 256, or 128 in the small form
        const int kvalid = KIND == kPairForward ? a.nz : (KIND == kPairInverse ? a.ny : a.nx);
        const int group = warp / GW, gw = warp % GW;
        const int q = kContig ? lane >> 3 : gw & 3;  // K column of 8 within the step
        const int row0 = kContig ? gw * 8 : (gw >> 2) * 32;
        const int row = row0 + (kContig ? lane & 7 : lane);
        constexpr int kRows = GW * 8;  // rows between a warp's tasks
        int mytasks = 0;  // tasks with rows of the operand
        while (mytasks < kTasks && row0 + mytasks * kRows < (int)rp)
            ++mytasks;
        const uint32_t soff = a.ring_off + (uint32_t)(q >> 1) * xchunk + (uint32_t)(q & 1) * rp * 16u +
                              (uint32_t)row * 16u;
        float pre[kTasks][8];
        const float *src = nullptr;  // this thread's row and K column of step 0
        int rows = 0;                // rows of the tile's operand that exist
        auto open_tile = [&](int i) {
            const Tile t = tile_at<KIND>(a, i);
            src = a.in + t.base + (kContig ? (long)(row * a.nz + q * 8)
                                           : (long)((uint32_t)row + (uint32_t)(q * 8) * ks));
            rows = KIND == kPairForward   ? a.ny
                   : KIND == kPairInverse ? a.nz
                                          : (int)min(128L, a.lines - t.row0);
            if (i + 1 < mine && group == 0) {
                const Tile n = tile_at<KIND>(a, i + 1);
                const float *p = a.in + n.base;
                if (KIND == kPairSpectral) {
                    const int l32 = (int)((min(128L, a.lines - n.row0) + 31) / 32);
                    for (int e = gw * 32 + lane; e < a.nx * 4; e += GW * 32)
                        if ((e & 3) < l32)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(
                                p + (uint32_t)(e >> 2) * ks + (e & 3) * 32));
                } else if (n.base != t.base) {
                    for (int e = gw * 32 + lane; e * 32 < a.ny * a.nz; e += GW * 32)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + e * 32));
                }
            }
        };
        auto load = [&](int st) {
            const int left = kvalid - st * 32 - q * 8;  // K of this column that exist
            const float *p = src + (kContig ? (uint32_t)(st * 32) : (uint32_t)(st * 32) * ks);
#pragma unroll
            for (int u = 0; u < kTasks; ++u) {
                if (u >= mytasks) continue;
                const int n = row + u * kRows < rows ? left : 0;
                if (kContig) {
                    const float *pu = p + (uint32_t)(u * kRows * a.nz);
                    if (VAR) {
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (4 * e < n) f = __ldg(reinterpret_cast<const float4 *>(pu) + e);
                            pre[u][4 * e] = f.x;
                            pre[u][4 * e + 1] = f.y;
                            pre[u][4 * e + 2] = f.z;
                            pre[u][4 * e + 3] = f.w;
                        }
                    } else {
#pragma unroll
                        for (int m = 0; m < 8; ++m) pre[u][m] = m < n ? __ldg(pu + m) : 0.0f;
                    }
                } else {
                    // plain loads: kPairSpectral stores over its own lines later in this kernel
                    const float *pu = p + u * kRows;
#pragma unroll
                    for (int m = 0; m < 8; ++m, pu += ks) pre[u][m] = m < n ? *pu : 0.0f;
                }
            }
        };
        // this group's steps: group, group + kGroups, ... of the CTA's sequence
        int li = 0, ls = group, slot = group;
        uint32_t ph = 1;  // phase of xfree: the first round finds every slot free
        bool ok = true, reused = false;
        auto normalise = [&]() {
            while (ls >= ns1) ls -= ns1, ++li;
        };
        normalise();
        if (li < mine) {
            open_tile(li);
            load(ls);
        }
        while (li < mine) {
            if (reused) {
                ok = umma::mbar_wait(&xfree[slot], ph, kPairWait);
                ok = !__any_sync(0xffffffffu, !ok || *err);
                if (!ok) break;
            }
            // the second chunk of the tile's last step may not exist
            if (2 * ls + (q >> 1) < a.nk1) {
                unsigned char *x = smem + soff + (uint32_t)slot * 2u * xchunk;
#pragma unroll
                for (int u = 0; u < kTasks; ++u)
                    if (u < mytasks && (kContig || row + u * kRows < (int)rp))
                        split8<PLANES>(x + u * kRows * 16, rp * 32u, pre[u]);
            }
            umma::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&xfull[slot]);
            slot += kGroups;
            if (slot >= a.ring) slot -= a.ring, ph ^= 1, reused = true;
            const int was = li;
            ls += kGroups;
            normalise();
            if (li < mine) {
                if (li != was) open_tile(li);
                load(ls);
            }
        }
        if (!ok) *err = 1;
    } else {
        // ---- epilogue warps --------------------------------------------------------------------
        const int quarter = warp & 3, part = (warp - NL) >> 2;
        constexpr int kParts = NE / 4;
        const uint32_t row = (uint32_t)quarter * 32u + (uint32_t)lane;
        const uint32_t tl = tmem + ((uint32_t)quarter * 32u << 16);
        const uint32_t tl2 = tl + (KIND == kPairSpectral ? (uint32_t)a.np1 : rp);
        const bool active = (uint32_t)quarter * 32u < tm;  // this warp has rows of the tile
        double part_cost = 0.0, part_raw = 0.0;
        DevState *st = nullptr;
        auto flush_costs = [&]() {
            if (KIND != kPairSpectral || !st) return;
            const double c = warp_sum(part_cost), r = a.want_raw ? warp_sum(part_raw) : 0.0;
            if (lane == 0) {
                atomicAdd(&st->lp_tr, c);
                if (a.want_raw) atomicAdd(&st->raw_reg, r);
            }
            part_cost = part_raw = 0.0;
        };
        float dnext[16];
        auto load_col = [&](const float *p, int c, bool valid, float *v) {
            uint32_t at = row + (uint32_t)(c * 16) * ks;
            const int left = valid ? a.nx - c * 16 : 0;
            if (left >= 16) {
#pragma unroll
                for (int m = 0; m < 16; ++m, at += ks) v[m] = __ldg(p + at);
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m, at += ks) v[m] = m < left ? __ldg(p + at) : 0.0f;
            }
        };
        const long ring = KIND == kPairInverse && a.ring_n > 1
                              ? (long)(a.st->sweep % a.ring_n) * a.ring_stride
                              : 0;
        Tile t = tile_at<KIND>(a, 0);
        if (KIND == kPairSpectral)
            load_col(a.D + t.row0, 2 * part, (long)t.row0 + row < a.lines, dnext);
        bool ok = true;
        for (int i = 0; i < mine; ++i) {
            const int bch = a.chain_comps ? t.comp / a.chain_comps : 0;
            const int cn = t.comp - bch * a.chain_comps;
            const Tile next = tile_at<KIND>(a, i + 1 < mine ? i + 1 : i);
            if (KIND == kPairSpectral && i + 1 < mine) {
                // the next tile's eigenvalues (and noise) on their way to L2: read from DRAM when
                // needed, each 16 of them cost a warp a microsecond
                const int lines128 = (int)((min(128L, a.lines - next.row0) + 31) / 32);
                for (int q = (int)(warp - NL) * 32 + lane; q < a.nx * 4; q += NE * 32) {
                    if ((q & 3) >= lines128) continue;
                    const uint32_t at = (uint32_t)(q >> 2) * ks + (uint32_t)(q & 3) * 32u;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.D + next.row0 + at));
                    if (VAR)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.noise + next.base + at));
                }
            }
            // ---- first accumulator -> second product's operand ----------------------------------
            ok = umma::mbar_wait(d1full, (uint32_t)i & 1u, kPairWait);
            ok = !__any_sync(0xffffffffu, !ok || *err);
            if (!ok) break;
            umma::fence_after_sync();
            auto publish = [&](int s) {  // step s of the second product's operand
                umma::fence_proxy_async_smem();
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) umma::mbar_arrive(&dready[s]);
            };
            if (KIND == kPairSpectral) {
                const bool valid = (long)t.row0 + row < a.lines;
                if (st != a.st + bch) {
                    flush_costs();
                    st = a.st + bch;
                }
                const double gamma = st->gamma[cn];
                const float gs2 = (float)(gamma * a.sigma2);
                const bool want_raw = a.want_raw && (st->sweep % a.every == 0);
                for (int g = part; g < ns2; g += kParts) {
                    // prior costs: FP32 partial sums over 32 coefficients, FP64 across
                    float ccost = 0.0f;
#pragma unroll 1
                    for (int c = 2 * g; c < min(2 * g + 2, a.nk2); ++c) {
                        float v[16], dcur[16], nz[16];
                        if (VAR) load_col(a.noise + t.base, c, valid, nz);
#pragma unroll
                        for (int m = 0; m < 16; ++m) dcur[m] = dnext[m];
                        // the next chunk's eigenvalues; after the last one, the next tile's first
                        const int cn1 = (c & 1) ? 2 * (g + kParts) : c + 1;
                        if (cn1 < a.nk2) load_col(a.D + t.row0, cn1, valid, dnext);
                        else load_col(a.D + next.row0, 2 * part,
                                      (long)next.row0 + row < a.lines, dnext);
                        umma::tmem_ld16(tl + (uint32_t)(c * 16), v);
                        // past the line's end the accumulator is zero, and so are D and the
                        // noise: no test per element
#pragma unroll
                        for (int m = 0; m < 16; ++m) {
                            const float Dv = dcur[m];
                            const float f = __fdividef(1.0f, fmaf(gs2, Dv, 1.0f));
                            // the roundings of the per-axis pass, whatever the compiler contracts
                            float val = __fmul_rn(v[m], f);
                            if (VAR) val = fmaf(sqrtf((float)a.sigma2 * f), nz[m], val);
                            ccost = fmaf(__fmul_rn(Dv, val), val, ccost);
                            v[m] = val;
                        }
                        unsigned char *x = smem + (uint32_t)c * dchunk + row * 16u;
                        split8<PLANES>(x, 128u * 32u, v);
                        split8<PLANES>(x + 128u * 16u, 128u * 32u, v + 8);
                    }
                    publish(g);
                    part_cost += 0.5 * gamma * (double)ccost;
                    if (want_raw) part_raw += a.eta2[cn] * a.rho_p * (double)ccost;
                }
            } else {
                for (int g = part; g < ns2; g += kParts) {
                    if (active) {
#pragma unroll 1
                        for (int c = 2 * g; c < min(2 * g + 2, a.nk2); ++c) {
                            float v[16];
                            umma::tmem_ld16(tl + (uint32_t)(c * 16), v);
                            if (row < tm) {
                                unsigned char *x = smem + (uint32_t)c * dchunk + row * 16u;
                                split8<PLANES>(x, tm * 32u, v);
                                split8<PLANES>(x + tm * 16u, tm * 32u, v + 8);
                            }
                        }
                    }
                    publish(g);
                }
            }

            // ---- second accumulator -> global ---------------------------------------------------
            ok = umma::mbar_wait(d2full, (uint32_t)i & 1u, kPairWait);
            ok = !__any_sync(0xffffffffu, !ok || *err);
            if (!ok) break;
            umma::fence_after_sync();
            float *o = a.out + t.base + ring;
            if (KIND == kPairInverse) {
                for (int mt = 0; mt * 128 < a.np2; ++mt) {
                    const int z = mt * 128 + (int)row;
                    if (mt * 128 + quarter * 32 >= a.nz) break;
                    const float pz = (float)z, px = (float)t.plane;
                    for (int c = part; c * 16 < (int)tm; c += kParts) {
                        float v[16];
                        umma::tmem_ld16(tl2 + (uint32_t)mt * tm + (uint32_t)(c * 16), v);
                        if (z >= a.nz) continue;
                        const int y0 = t.row0 + c * 16;
                        const int left = min(a.ny - y0, (int)tm - c * 16);
                        uint32_t at = (uint32_t)(y0 * a.nz + z);
                        if (a.xpos) {
                            const float *xp = a.xpos + (t.base - (long)t.comp * a.V) + (long)cn * a.V;
                            float pos[16];
#pragma unroll
                            for (int m = 0; m < 16; ++m)
                                pos[m] = m < left ? __ldg(xp + (at + (uint32_t)(m * a.nz))) : 0.0f;
#pragma unroll
                            for (int m = 0; m < 16; ++m) v[m] += pos[m];
                        } else {
                            const float p0 = cn == 2 ? pz : (cn == 0 ? px : (float)y0);
                            const float dp = cn == 1 ? 1.0f : 0.0f;  // whole numbers: exact
#pragma unroll
                            for (int m = 0; m < 16; ++m) v[m] += fmaf((float)m, dp, p0);
                        }
                        if (left >= 16) {
#pragma unroll
                            for (int m = 0; m < 16; ++m, at += (uint32_t)a.nz) o[at] = v[m];
                        } else {
#pragma unroll
                            for (int m = 0; m < 16; ++m, at += (uint32_t)a.nz)
                                if (m < left) o[at] = v[m];
                        }
                    }
                }
            } else if (active) {
                // lanes: kz of the tile (forward), lines (spectral); columns: ky, x
                const int cols = KIND == kPairForward ? a.ny : a.nx;
                const bool valid = row < tm && (KIND == kPairForward
                                                    ? t.row0 + (int)row < a.nz
                                                    : (long)t.row0 + row < a.lines);
                const uint32_t off = (KIND == kPairForward ? (uint32_t)t.row0 : 0u) + row;
                for (int c = part; c * 16 < cols; c += kParts) {
                    float v[16];
                    umma::tmem_ld16(tl2 + (uint32_t)(c * 16), v);
                    if (!valid) continue;
                    uint32_t at = off + (uint32_t)(c * 16) * ks;
                    const int left = cols - c * 16;
                    if (left >= 16) {
#pragma unroll
                        for (int m = 0; m < 16; ++m, at += ks) o[at] = v[m];
                    } else {
#pragma unroll
                        for (int m = 0; m < 16; ++m, at += ks)
                            if (m < left) o[at] = v[m];
                    }
                }
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(d2free);
            t = next;
        }
        if (!ok) *err = 1;
        flush_costs();
    }

    // ---- teardown: after an error, let every tcgen05 op still in flight finish (bounded) ----
    __syncthreads();
    if (*s_err && tid == kMma * 32) {
        umma::commit(drain);
        umma::mbar_wait(drain, 0, kPairWait);
        if (a.st) atomicOr(&a.st->flags, (unsigned)kFlagTensorTimeout);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == NL) umma::tmem_dealloc(tmem, a.ncols);
}

int pad16(int n) { return (n + 15) / 16 * 16; }

// the shapes of one launch; smem 0: not supported
struct PairShape {
    int rp, tm, tiles, nk1, nk2, mats, ring, nl, ne;
    uint32_t ring_off, mat_off, mat_slot, bar_off, ncols;
    size_t smem;
    long ctas;  // tiles per component
};

PairShape pair_shape(PairKind kind, int nx, int ny, int nz, int planes, int ncomp,
                     bool sample) {
    PairShape p{};
    if (nx > kMaxAxis || ny > kMaxAxis || nz > kMaxAxis) return p;
    const uint32_t pb = (uint32_t)planes * 32u;
    int d1cols, np2, mrows1;
    if (kind == kPairSpectral) {
        p.rp = p.tm = 128;
        p.tiles = ceil_div((long)ny * nz, 128);
        p.ctas = p.tiles;
        p.nk1 = pad16(nx) / 16;
        d1cols = np2 = mrows1 = pad16(nx);
    } else {
        // the tiled output axis (forward: kz, inverse: y) in equal tiles of at most 128
        const int n = kind == kPairForward ? nz : ny;
        p.tiles = ceil_div(n, 128);
        p.tm = pad16(ceil_div(n, p.tiles));
        p.ctas = (long)nx * p.tiles;
        p.rp = pad16(kind == kPairForward ? ny : nz);
        p.nk1 = pad16(kind == kPairForward ? nz : ny) / 16;
        d1cols = np2 = p.rp;
        mrows1 = p.tm;
    }
    p.nk2 = d1cols / 16;
    const uint32_t d2cols =
        kind == kPairInverse ? (uint32_t)(ceil_div(np2, 128) * p.tm) : (uint32_t)np2;
    p.ncols = 32;
    while (p.ncols < (uint32_t)d1cols + d2cols) p.ncols <<= 1;
    if (p.ncols > 512) return p;
    const uint32_t xslot = 2 * pb * p.rp, dbuf = pb * p.tm * p.nk2;
    p.mat_slot = 2 * pb * std::max(mrows1, np2);
    p.ring_off = dbuf;
    const uint32_t slack = kind == kPairSpectral ? 0 : kSlack;
    const size_t bars = (size_t)(2 * kMaxRing + kMaxSteps + 2 * kMaxMat + 4) * 8 + 64;
    const size_t fixed = (size_t)dbuf + slack + bars;
    auto total = [&](int ring, int mats) {
        return fixed + (size_t)ring * xslot + (size_t)mats * p.mat_slot;
    };
    // Two CTAs per SM where their tables and accumulators fit and there are tiles for them (a group
    // of four load warps covers 128 rows in its four tasks), else one.  Load + epilogue warps:
    //   forward, inverse  8 + 4 of two CTAs, 16 + 8 of one;
    //   spectral          4 + 4 of two CTAs (14.7 us at 91x109x91; 4 + 12 of one 19.3, 8 + 4 of two
    //                     16.9, which spill), 8 + 12 of one (55 us at 160x192x160; 4 + 12 58);
    //   with the noise    4 + 12 of one (424 us per sweep of 32 chains at 96^3; 8 + 12 503 and
    //                     8 + 8 526, with spills; 4 + 4 of two the same 423).
    const bool two = !sample && p.rp <= 128 && p.ncols <= 256 && total(2, 2) <= 112 * 1024 &&
                     p.ctas * ncomp > 148;
    const size_t limit = two ? 112 * 1024 : 226 * 1024;
    if (kind == kPairSpectral) {
        p.nl = two || sample ? 4 : 8;
        p.ne = two ? 4 : 12;
    } else {
        p.nl = two ? 8 : 16;
        p.ne = two ? 4 : 8;
    }
    p.ring = 2;
    p.mats = 2;
    if (total(p.ring, 2) > limit) return p;
    // what is left goes to the rings in turn
    const int most = std::max(p.ring, std::min(kMaxRing, p.nk1));
    while (true) {
        const bool more_ring = p.ring < most && total(p.ring + 1, p.mats) <= limit;
        const bool more_mats = p.mats < kMaxMat && total(p.ring, p.mats + 1) <= limit;
        if (more_mats && (p.mats < p.ring || !more_ring)) ++p.mats;
        else if (more_ring) ++p.ring;
        else break;
    }
    p.mat_off = p.ring_off + p.ring * xslot;
    p.bar_off = p.mat_off + p.mats * p.mat_slot + slack;
    p.smem = total(p.ring, p.mats);
    return p;
}

template <int KIND, int PLANES, int NL, int NE, bool VAR>
void launch(const PairArgs &a, const PairShape &p, cudaStream_t s) {
    auto *fn = pair_kernel<KIND, PLANES, NL, NE, VAR>;
    constexpr int per_sm = NE == 4 ? 2 : 1;
    // at most per_sm CTAs on an SM, whatever would fit: tcgen05.alloc of a surplus CTA would wait
    const size_t smem = std::max(p.smem, (size_t)(per_sm == 1 ? 115 : 77) * 1024);
    BINDER_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    BINDER_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared));
    int dev = 0, sms = 148;
    BINDER_CUDA(cudaGetDevice(&dev));
    BINDER_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long grid = std::min(a.total, (long)sms * per_sm);
    count_launch(), fn<<<(unsigned)grid, (NL + NE + 2) * 32, smem, s>>>(a);
    BINDER_CUDA(cudaGetLastError());
}

template <int KIND, int PLANES, bool VAR>
void launch_kind(const PairArgs &a, const PairShape &p, cudaStream_t s) {
    if constexpr (KIND == kPairSpectral) {
        if constexpr (VAR) {
            launch<KIND, PLANES, 4, 12, VAR>(a, p, s);
        } else {
            if (p.ne == 12) launch<KIND, PLANES, 8, 12, VAR>(a, p, s);
            else launch<KIND, PLANES, 4, 4, VAR>(a, p, s);
        }
    } else {
        if (p.ne == 8) launch<KIND, PLANES, 16, 8, VAR>(a, p, s);
        else launch<KIND, PLANES, 8, 4, VAR>(a, p, s);
    }
}

template <int PLANES>
void launch_planes(PairKind kind, const PairArgs &a, const PairShape &p, cudaStream_t s) {
    switch (kind) {
        case kPairForward:
            if (a.nz % 4 == 0) launch_kind<kPairForward, PLANES, true>(a, p, s);
            else launch_kind<kPairForward, PLANES, false>(a, p, s);
            break;
        case kPairSpectral:
            if (a.sample) launch_kind<kPairSpectral, PLANES, true>(a, p, s);
            else launch_kind<kPairSpectral, PLANES, false>(a, p, s);
            break;
        case kPairInverse: launch_kind<kPairInverse, PLANES, false>(a, p, s); break;
    }
}

}  // namespace

bool pair_supported(int nx, int ny, int nz, int planes) {
    // (the one-CTA forms, which the two-CTA forms are smaller than)
    if (nz == 1) return pair_shape(kPairSpectral, nx, ny, nz, planes, 1, false).smem > 0;
    for (PairKind k : {kPairForward, kPairSpectral, kPairInverse})
        if (pair_shape(k, nx, ny, nz, planes, 1, false).smem == 0) return false;
    return true;
}

void launch_pair_pass(const AxisArgs<float> &b, PairKind kind, int nx, int ny, int nz,
                      const UmmaMatrix &M1, const UmmaMatrix &M2, int ncomp, int planes,
                      cudaStream_t s) {
    BINDER_CHECK(planes == 1 || planes == 2, "planes must be 1 (one product) or 2 (split)");
    const PairShape p = pair_shape(kind, nx, ny, nz, planes, ncomp, kind == kPairSpectral && b.sample);
    BINDER_CHECK(p.smem > 0, "the volume does not fit the paired transform passes");
    const int n1 = kind == kPairForward ? nz : (kind == kPairSpectral ? nx : ny);
    const int n2 = kind == kPairForward ? ny : (kind == kPairSpectral ? nx : nz);
    BINDER_CHECK(M1.n == n1 && M2.n == n2, "matrix / axis length mismatch");
    BINDER_CHECK(p.ctas * ncomp < (1L << 31), "transform grid too large");
    BINDER_CHECK(!b.sample || kind != kPairSpectral || b.noise, "sampling needs the prior noise");
    PairArgs a{};
    a.in = b.in; a.out = b.out; a.V = b.comp_stride;
    a.m1 = reinterpret_cast<const unsigned char *>(M1.dev16);
    a.m2 = reinterpret_cast<const unsigned char *>(M2.dev16);
    a.np1 = M1.Npad; a.np2 = M2.Npad; a.nk1 = p.nk1; a.nk2 = p.nk2;
    a.nx = nx; a.ny = ny; a.nz = nz; a.lines = (long)ny * nz;
    a.rp = p.rp; a.tm = p.tm; a.tiles = p.tiles; a.mats = p.mats; a.ring = p.ring;
    a.ctas = p.ctas; a.total = p.ctas * ncomp; a.ring_off = p.ring_off;
    a.mat_off = p.mat_off; a.mat_slot = p.mat_slot; a.bar_off = p.bar_off; a.ncols = p.ncols;
    a.D = b.D; a.st = b.st; a.sigma2 = b.sigma2; a.sample = b.sample; a.want_raw = b.want_raw;
    a.every = b.every < 1 ? 1 : b.every; a.noise = b.noise; a.rho_p = b.rho_p;
    for (int i = 0; i < 3; ++i) a.eta2[i] = b.eta2[i];
    a.xpos = b.xpos; a.dims = b.dims; a.comp0 = b.comp0; a.chain_comps = b.chain_comps;
    a.ring_n = b.ring_n; a.ring_stride = b.ring_stride; a.skip = b.skip;
    if (planes == 2) launch_planes<2>(kind, a, p, s);
    else launch_planes<1>(kind, a, p, s);
}

}  // namespace binder
