// The DCT-prior M-step of a small 2D image (nx, ny <= 128) in one launch, for the images where
// the separate passes are each a couple of CTAs' latency.  One thread-block cluster of G CTAs
// per component:
//   1. CTA q owns the rows [q R, (q + 1) R) (R = ceil(nx / G), up to a multiple of 4): forward
//      DCT along y;
//   2. cluster barrier; CTA q gathers the columns [q W, (q + 1) W) (W from ny like R) of every
//      row from the other CTAs' shared memory (distributed shared memory), forward DCT along x,
//      prior scaling 1 / (1 + gamma sigma^2 D) [+ noise] with the costs, inverse DCT along x;
//   3. cluster barrier; CTA q gathers its rows back, inverse DCT along y, adds the pixel
//      positions and stores.
// Each product is out[k] = sum_j MT[j][k] in[j] with the pass matrix staged transposed in
// shared memory (lanes take consecutive k: conflict-free rows), FP32 FMA; the epilogue is that
// of the CUDA-core passes (transform.cu): the same scaling, noise stream and FP64 costs.
//
// The kernel is bound by what shared memory can hand to the registers (128 bytes a cycle per SM,
// broadcast or not) and by the latencies between its barriers.  Both operands of a product are
// read as vectors: the slab stands [j][q], and its rows and columns come over distributed shared
// memory four floats at a time into that form.  D is in registers before the product that needs
// it, and the first loads are issued before the skip flag is looked at.  At 128 x 128 a launch
// takes 13.9 us with clusters of 16, tiles of 2 x 2, and 20.4 us with clusters of 8, tiles of
// 4 x 2 (it was 41 us with clusters of 8, a scalar slab and the D loads between the stores).
// Clusters of 16 are the rule; 8 is for a device or a partition that cannot place 16 on one
// cluster of SMs.  Other tiles measured: 4 x 2 with 128 threads 16.8 us (16), 4 x 4 21.0 us (8).
#include <cooperative_groups.h>

#include "mstep2d.cuh"

namespace cg = cooperative_groups;

namespace binder {

namespace {

constexpr int kM2dThreads = 256;

// the split for a cluster of G CTAs per component
template <int G>
struct Split {
    static constexpr int kSlab = (kM2dMaxN + G - 1) / G;  // most rows / columns per CTA
    // floats between the [j] rows of a [j][q] slab (16-byte rows, and a transposing store of
    // consecutive j meets 8 banks)
    static constexpr int kStride = kSlab + 4;
    // a thread's tile of a product: kPT of up to 128 outputs p and kQT of up to kSlab outputs q;
    // a warp covers 16 kPT p (16 lanes) x 2 kQT q (2 half-warps)
    static constexpr int kPT = G == 16 ? 2 : 4, kQT = 2;
    static constexpr int kPWarps = kM2dMaxN / (16 * kPT);
    static_assert(kM2dThreads / 32 / kPWarps * 2 * kQT == kSlab, "the tiles cover 128 x kSlab");
    static constexpr size_t kSmem = (size_t)(2 * kM2dMaxN * kM2dMaxN + 2 * kM2dMaxN * kStride +
                                             2 * kSlab * kM2dMaxN) * sizeof(float);
};

struct M2dArgs {
    AxisArgs<float> a;
    const float *r;
    float *d;
    int nx, ny;
    const float *Fx, *Ix, *Fy, *Iy;
};

// start copying the n x n matrix M into shared memory, rows padded to a multiple of 4 floats
// (cp.async: 16-byte pieces, or 4-byte ones where a row of M is not a multiple of 16 bytes; M and
// ms are 16-byte aligned); stage_wait() completes it
__device__ __forceinline__ void stage_async(float *ms, const float *M, int n) {
    if ((n & 3) == 0) {
        for (int f = threadIdx.x; f < n * n / 4; f += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(ms + 4 * f)),
                         "l"(M + 4 * f)
                         : "memory");
    } else {
        const int stride = (n + 3) & ~3;
        const int lane = threadIdx.x & 31;
        for (int j = threadIdx.x >> 5; j < n; j += blockDim.x >> 5)
            for (int k = lane; k < n; k += 32)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(ms + j * stride + k)),
                             "l"(M + j * n + k)
                             : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void stage_wait() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

template <int G>
struct Tile {
    int p0, q0;
    __device__ __forceinline__ Tile() {
        using S = Split<G>;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        p0 = S::kPT * (16 * (warp % S::kPWarps) + (lane & 15));
        q0 = S::kQT * (2 * (warp / S::kPWarps) + (lane >> 4));
    }
};

template <int N>
__device__ __forceinline__ void load_vec(float (&v)[N], const float *p) {
    static_assert(N == 2 || N == 4, "a vector load");
    if constexpr (N == 4) {
        const float4 w = *reinterpret_cast<const float4 *>(p);
        v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
    } else {
        const float2 w = *reinterpret_cast<const float2 *>(p);
        v[0] = w.x; v[1] = w.y;
    }
}

// out(p, q) = sum_{j < len} X[j xs + p] Y[j kStride + q], j ascending, for the tile's outputs
// with p < P and q < Q; xs is a multiple of 4
template <int G, int kQT, int kPT>
__device__ __forceinline__ void product(const Tile<G> &t, int P, int Q, int len, const float *X,
                                        int xs, const float *Y, float (&acc)[kQT][kPT]) {
#pragma unroll
    for (int q = 0; q < kQT; ++q)
#pragma unroll
        for (int e = 0; e < kPT; ++e) acc[q][e] = 0.0f;
    if (t.p0 >= P || t.q0 >= Q) return;  // no output here (no barrier follows inside)
    const float *x = X + t.p0, *y = Y + t.q0;
#pragma unroll 16
    for (int j = 0; j < len; ++j) {
        float xv[kPT], yv[kQT];
        load_vec(xv, x + j * xs);
        load_vec(yv, y + j * Split<G>::kStride);
#pragma unroll
        for (int q = 0; q < kQT; ++q)
#pragma unroll
            for (int e = 0; e < kPT; ++e) acc[q][e] = fmaf(xv[e], yv[q], acc[q][e]);
    }
}

// the tile as rows of p: dst[q][p], 128 floats to a row (outputs past P write padding)
template <int G, int kQT, int kPT>
__device__ __forceinline__ void store_rows(const Tile<G> &t, int P, int Q, float *dst,
                                           const float (&acc)[kQT][kPT]) {
    if (t.p0 >= P) return;
#pragma unroll
    for (int q = 0; q < kQT; ++q) {
        if (t.q0 + q >= Q) continue;
        float *d = dst + (t.q0 + q) * kM2dMaxN + t.p0;
        if constexpr (kPT == 4)
            *reinterpret_cast<float4 *>(d) = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
        else
            *reinterpret_cast<float2 *>(d) = make_float2(acc[q][0], acc[q][1]);
    }
}

// slab[j][0 .. count) (j < len) from the CTAs' rows: CTA o holds rows [o step, (o + 1) step) of
// the transposed order as rows[j - o step][at + q]; four floats per load.  Reads up to 3 floats
// past `count` inside the row's 128, which no stored output uses.
template <int G>
__device__ __forceinline__ void gather(cg::cluster_group &cluster, float *slab, float *rows,
                                       int len, int step, int at, int count) {
    const int quads = (count + 3) >> 2;
    constexpr int kQuads = Split<G>::kSlab / 4, kStride = Split<G>::kStride;
    const int quad = threadIdx.x % kQuads;  // kQuads threads to a row
    if (quad >= quads) return;
    constexpr int kRows = kM2dThreads / kQuads;
    float4 v[kM2dMaxN / kRows];
#pragma unroll
    for (int u = 0; u < kM2dMaxN / kRows; ++u) {
        const int j = threadIdx.x / kQuads + u * kRows;
        if (j < len) {
            const int owner = j / step;
            const float *src = cluster.map_shared_rank(rows, owner);
            v[u] = *reinterpret_cast<const float4 *>(src + (j - owner * step) * kM2dMaxN + at +
                                                     4 * quad);
        }
    }
#pragma unroll
    for (int u = 0; u < kM2dMaxN / kRows; ++u) {
        const int j = threadIdx.x / kQuads + u * kRows;
        if (j < len) *reinterpret_cast<float4 *>(slab + j * kStride + 4 * quad) = v[u];
    }
}

template <int G>
__global__ void __cluster_dims__(G, 1, 1) __launch_bounds__(kM2dThreads)
    mstep2d_kernel(const M2dArgs p) {
    constexpr int kSlab = Split<G>::kSlab, kStride = Split<G>::kStride;
    constexpr int kPT = Split<G>::kPT, kQT = Split<G>::kQT;
    const AxisArgs<float> &a = p.a;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) float sm[];
    const int nx = p.nx, ny = p.ny;
    // rows and columns per CTA, multiples of 4 so that a slab's pieces are whole vectors
    const int R = ((nx + G - 1) / G + 3) & ~3, W = ((ny + G - 1) / G + 3) & ~3;
    const int sx = (nx + 3) & ~3, sy = (ny + 3) & ~3;  // row strides of the staged matrices
    float *ms0 = sm;                           // [n][stride] pass matrices (transposed: [j][k]),
    float *ms1 = ms0 + kM2dMaxN * kM2dMaxN;    // double-buffered
    float *slab = ms1 + kM2dMaxN * kM2dMaxN;   // [j][q]: this CTA's rows or columns, transposed
    float *slab2 = slab + kM2dMaxN * kStride;
    float *rowB = slab2 + kM2dMaxN * kStride;  // [xl][ky], read by the other CTAs
    float *colA = rowB + kSlab * kM2dMaxN;         // [yl][x], read by the other CTAs
    __shared__ double red[32];
    const int q = (int)cluster.block_rank();
    const int comp = (int)blockIdx.y;
    const long V = a.comp_stride;
    const int x0 = q * R, nr = max(0, min(R, nx - x0));  // my rows
    const int y0 = q * W, nw = max(0, min(W, ny - y0));  // my columns
    const int tid = threadIdx.x;
    const Tile<G> t;
    float acc[kQT][kPT];

    // ---- 1. forward DCT along y of my rows: rowB[x][ky] = sum_y Fy[ky][y] r[x][y] --------------
    // the first loads are on their way before the skip flag is looked at
    stage_async(ms0, p.Iy, ny);  // Iy[y][ky] = Fy[ky][y]
    {
        const float *src = p.r + comp * V + (long)x0 * ny;
        // warp -> rows, lanes -> y: coalesced loads, transposed on the way
        const int lane = tid & 31, warp = tid >> 5;
        constexpr int kWarps = kM2dThreads / 32;
        float v[kSlab / kWarps][kM2dMaxN / 32];
#pragma unroll
        for (int i = 0; i < kSlab / kWarps; ++i)
#pragma unroll
            for (int c = 0; c < kM2dMaxN / 32; ++c) {
                const int xl = warp + i * kWarps, y = lane + 32 * c;
                v[i][c] = xl < nr && y < ny ? __ldg(src + xl * ny + y) : 0.0f;
            }
        if (a.skip && *a.skip) {  // the same decision in every CTA of the cluster
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            return;
        }
#pragma unroll
        for (int i = 0; i < kSlab / kWarps; ++i)
#pragma unroll
            for (int c = 0; c < kM2dMaxN / 32; ++c)
                slab[(lane + 32 * c) * kStride + warp + i * kWarps] = v[i][c];
    }
    const double g = a.st->gamma[comp];
    const uint32_t sweep = (uint32_t)a.st->sweep;
    const bool want_raw = a.want_raw && (a.st->sweep % a.every == 0);
    stage_wait();
    stage_async(ms1, p.Ix, nx);  // Ix[x][kx] = Fx[kx][x], in flight during the y pass
    // p = ky (X = Iy rows y), q = xl
    product(t, ny, nr, ny, ms0, sy, slab, acc);
    store_rows(t, ny, nr, rowB, acc);
    // the prior eigenvalues of this thread's coefficients (kx, ky), flat index kx ny + ky
    float Dv[kQT][kPT];
#pragma unroll
    for (int qq = 0; qq < kQT; ++qq)
#pragma unroll
        for (int e = 0; e < kPT; ++e)
            Dv[qq][e] = t.p0 + e < nx && t.q0 + qq < nw
                            ? __ldg(a.D + (long)(t.p0 + e) * ny + y0 + t.q0 + qq)
                            : 0.0f;
    cluster.sync();  // every CTA's rowB is complete

    // ---- 2. my columns of every row, forward x, scaling, inverse x --------------------------
    gather<G>(cluster, slab, rowB, nx, R, y0, nw);
    stage_wait();                // Ix, and the slab; every thread is done with ms0 (the barrier)
    stage_async(ms0, p.Fx, nx);  // inverse: x = sum_kx Fx[kx][x] c[kx]
    double part_cost = 0.0, part_raw = 0.0;
    {
        const float gs2 = (float)(g * a.sigma2);
        // p = kx (X = Ix rows x), q = yl
        product(t, nx, nw, nx, ms1, sx, slab, acc);
        float f[kQT][kPT];
#pragma unroll
        for (int qq = 0; qq < kQT; ++qq)
#pragma unroll
            for (int e = 0; e < kPT; ++e) {
                f[qq][e] = 1.0f / (1.0f + gs2 * Dv[qq][e]);
                if (!a.sample) acc[qq][e] = acc[qq][e] * f[qq][e];
            }
        if (a.sample)
#pragma unroll
            for (int qq = 0; qq < kQT; ++qq)
#pragma unroll
                for (int e = 0; e < kPT; ++e) {
                    if (t.p0 + e >= nx || t.q0 + qq >= nw) continue;
                    const long i = (long)(t.p0 + e) * ny + (y0 + t.q0 + qq);
                    acc[qq][e] = fmaf(sqrtf((float)a.sigma2 * f[qq][e]),
                                      dct_prior_normal(a.seed, (uint32_t)i, sweep, a.chain, comp),
                                      __fmul_rn(acc[qq][e], f[qq][e]));
                }
#pragma unroll
        for (int e = 0; e < kPT; ++e)
#pragma unroll
            for (int qq = 0; qq < kQT; ++qq) {
                if (t.p0 + e >= nx || t.q0 + qq >= nw) continue;
                const float v = acc[qq][e];
                const double v2 = (double)v * (double)v;
                part_cost += 0.5 * g * (double)Dv[qq][e] * v2;
                if (want_raw) part_raw += a.eta2[comp] * a.rho_p * (double)Dv[qq][e] * v2;
                slab2[(t.p0 + e) * kStride + t.q0 + qq] = v;
            }
    }
    stage_wait();                // Fx, and slab2 complete
    stage_async(ms1, p.Fy, ny);  // inverse: y = sum_ky Fy[ky][y] c[ky]
    // p = x (X = Fx rows kx), q = yl
    product(t, nx, nw, nx, ms0, sx, slab2, acc);
    store_rows(t, nx, nw, colA, acc);
    cluster.sync();  // every CTA's colA is complete (and nobody reads rowB any more)

    // ---- 3. my rows back, inverse y, positions -----------------------------------------------
    gather<G>(cluster, slab, colA, ny, W, x0, nr);
    stage_wait();  // Fy, and the slab
    // p = y (X = Fy rows ky), q = xl
    product(t, ny, nr, ny, ms1, sy, slab, acc);
#pragma unroll
    for (int qq = 0; qq < kQT; ++qq)
#pragma unroll
        for (int e = 0; e < kPT; ++e) {
            const int xl = t.q0 + qq, y = t.p0 + e;
            if (xl >= nr || y >= ny) continue;
            const long i = (long)(x0 + xl) * ny + y;
            const float xv =
                a.xpos ? a.xpos[comp * V + i] : (comp == 0 ? (float)(x0 + xl) : (float)y);
            p.d[comp * V + i] = acc[qq][e] + xv;
        }
    const double sc = block_sum(part_cost, red);
    if (tid == 0) atomicAdd(&a.st->lp_tr, sc);
    if (a.want_raw) {
        const double sr = block_sum(part_raw, red);
        if (tid == 0) atomicAdd(&a.st->raw_reg, sr);
    }
    cluster.sync();  // no CTA leaves while another may still read its shared memory
}

template <int G>
void configure() {
    BINDER_CUDA(cudaFuncSetAttribute(mstep2d_kernel<G>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)Split<G>::kSmem));
    if (G > 8)
        BINDER_CUDA(cudaFuncSetAttribute(mstep2d_kernel<G>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

}  // namespace

int mstep2d_cluster(bool portable) {
    configure<8>();
    if (portable) return 8;
    if (cudaFuncSetAttribute(mstep2d_kernel<16>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess) {
        cudaGetLastError();
        return 8;
    }
    configure<16>();
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(16, 2, 1);
    c.blockDim = dim3(kM2dThreads, 1, 1);
    c.dynamicSmemBytes = Split<16>::kSmem;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 16;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    c.attrs = &attr;
    c.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, mstep2d_kernel<16>, &c) != cudaSuccess) {
        cudaGetLastError();
        return 8;
    }
    return clusters >= 1 ? 16 : 8;
}

void launch_mstep2d(const AxisArgs<float> &a, const float *r, float *d, int nx, int ny,
                    const float *Fx, const float *Ix, const float *Fy, const float *Iy,
                    int cluster, cudaStream_t s) {
    BINDER_CHECK(nx >= 1 && ny >= 1 && nx <= kM2dMaxN && ny <= kM2dMaxN,
                 "the fused 2D M-step needs nx, ny <= 128");
    BINDER_CHECK(cluster == 8 || cluster == 16, "the fused 2D M-step's clusters have 8 or 16 CTAs");
    M2dArgs p{a, r, d, nx, ny, Fx, Ix, Fy, Iy};
    if (cluster == 16)
        count_launch(), mstep2d_kernel<16>
            <<<dim3(16, 2, 1), kM2dThreads, Split<16>::kSmem, s>>>(p);
    else
        count_launch(), mstep2d_kernel<8>
            <<<dim3(8, 2, 1), kM2dThreads, Split<8>::kSmem, s>>>(p);
    BINDER_CUDA(cudaGetLastError());
}

}  // namespace binder
