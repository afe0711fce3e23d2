// FP64 Hartley transforms H[k] = sum_j x[j] cas(2 pi j k / n) along one axis, on the FP64 matrix
// instructions.
//
// Folding: with e_j = x_j + x_{n-j} and o_j = x_j - x_{n-j} (j = 1 .. n/2; x_0, and x_{n/2} of an
// even n, in e alone), C_k = sum_j e_j cos(2 pi j k / n) and S_k = sum_j o_j sin(2 pi j k / n) for
// k = 0 .. n/2 give H[k] = C_k + S_k and H[n-k] = C_k - S_k: two products of (n/2)^2 instead of one
// of n^2, half the operations.
//
// A CTA folds its 32 (or 8) lines into shared memory (e and o, [j][32] with a pitch of 36 doubles, or
// [j][8] with 12: the four rows of a fragment are 8 banks apart), and each warp computes its 8-row
// tiles of both products for all the lines with mma.m8n8k4 (FP64 in, FP64 FMA accumulation), the
// matrices coming from global memory through L1.  kHartleyPoisson folds the scaled coefficients
// straight from the accumulators -- a thread holds k and n - k of its lines -- and transforms again,
// so the spectrum is never stored.
//
// Bound: the FP64 pipe (0.5 n FMA per element and pass; 5.1 GFLOP per pass at 160x192x160, 0.14 ms at
// 36 TFLOP/s).  Three components at 160x192x160, z / y / x with the Poisson scaling / y / z back:
// 0.18 / 0.21 / 0.34 / 0.21 / 0.19 ms, where a 64-line register-blocked FMA kernel of the unfolded
// matrix took 0.6 / 0.95 / 0.95 / 0.95 / 0.6 (one CTA of eight warps per SM, its staging not
// overlapped, a division per staged element).
//
// A CTA of 32 lines has a warp for every two 8-row tiles of the halves (17 tiles at most, at n = 256),
// so no warp idles but for an odd last tile, and two or three CTAs share an SM, one's folding
// overlapping another's products.  Four warps with three or four tiles each took 0.21 / 0.29
// / 0.34 / 0.29 / 0.21: 13 tiles leave three of 16 slots empty.  96 registers are what keeps three CTAs of
// six warps (or of seven) on an SM; with 128 the passes are 10 to 15 % slower, with 80 (three CTAs
// asked for of seven warps) 30 %.  Where 32 lines would leave SMs without a CTA, a CTA has 8 lines
// and a warp per tile (two components at 128x128, y / x with the Poisson scaling / y back: 4.4 /
// 6.8 / 4.4 us, against 14.6 / 29.0 / 14.8 with 32 lines).
#include <cmath>
#include <vector>

#include "hartley.cuh"
#include "layout.cuh"

namespace binder {
namespace {

// LT: 8-line tiles of a CTA (4 or 1)
template <int LT>
constexpr int kLinesH = 8 * LT;
template <int LT>
constexpr int kPitchH = 8 * LT + 4;  // doubles per row of e / o

struct HArgs {
    HartleyArgs a;
    const double *cs, *sn;
    int n, cols, tiles;  // tiles: 8-row tiles of the halves
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// both products of this warp's tiles: cC = cos e, cS = sin o
template <int U, int LT>
__device__ __forceinline__ void products(const HArgs &h, const double *E, const double *O,
                                         double (&cC)[U][LT][2], double (&cS)[U][LT][2], int warp,
                                         int nw, int lane) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int t = 0; t < LT; ++t) cC[u][t][0] = cC[u][t][1] = cS[u][t][0] = cS[u][t][1] = 0.0;
    const int ar = lane >> 2, ak = lane & 3;
    const double *pc[U], *ps[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        // tiles past the last one repeat it: their results are not stored
        const int m = min(warp + nw * u, h.tiles - 1);
        pc[u] = h.cs + (long)(m * 8 + ar) * h.cols + ak;
        ps[u] = h.sn + (long)(m * 8 + ar) * h.cols + ak;
    }
    double a0[U], a1[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a0[u] = __ldg(pc[u]), a1[u] = __ldg(ps[u]);
    for (int j = 0; j < h.cols; j += 4) {
        double n0[U], n1[U];  // the next step's matrix fragments, in flight during this one
        const int jn = j + 4 < h.cols ? j + 4 : j;
#pragma unroll
        for (int u = 0; u < U; ++u) n0[u] = __ldg(pc[u] + jn), n1[u] = __ldg(ps[u] + jn);
        const double *e = E + (j + ak) * kPitchH<LT> + ar, *o = O + (j + ak) * kPitchH<LT> + ar;
#pragma unroll
        for (int t = 0; t < LT; ++t) {
            const double be = e[t * 8], bo = o[t * 8];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                dmma(cC[u][t], a0[u], be);
                dmma(cS[u][t], a1[u], bo);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) a0[u] = n0[u], a1[u] = n1[u];
    }
}

// U: 8-row tiles per warp; W: warps of a CTA at most (a warp for every U tiles); CTAS: to an SM
template <int U, int MODE, int LT, int W, int CTAS>
__global__ void __launch_bounds__(32 * W, CTAS)
    hartley_kernel(const HArgs h) {
    constexpr int kLines = kLinesH<LT>, kPitch = kPitchH<LT>;
    extern __shared__ __align__(16) double sm[];
    double *E = sm, *O = sm + (long)h.cols * kPitch;
    const HartleyArgs &a = h.a;
    const int n = h.n, half = n >> 1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    const int comp = blockIdx.y;
    const double *in = a.in + comp * a.V;
    double *out = a.out + comp * a.V;
    const bool contig = a.s == 1;
    long base;  // first element of the tile
    int nl;     // lines of the tile
    long t0 = 0;
    if (contig) {
        const long l0 = (long)blockIdx.x * kLines;
        nl = (int)min((long)kLines, a.outer - l0);
        base = l0 * n;
    } else {
        const long tiles = (a.s + kLines - 1) / kLines;
        const long o = blockIdx.x / tiles;
        t0 = (blockIdx.x - o * tiles) * kLines;
        nl = (int)min((long)kLines, a.s - t0);
        base = o * n * a.s + t0;
    }
    const long js = contig ? 1 : a.s, ls = contig ? n : 1;  // strides of j and of the lines
    // ---- fold: contiguous lines 8 j x 4 lines per warp instruction (64-byte segments), strided
    // ones all the neighbouring lines (x 4 j for 8 lines)
    const int wj = contig ? 8 : 32 / kLines;  // j per warp instruction
    const int lj = contig ? lane & 7 : lane / kLines, ll = contig ? lane >> 3 : lane % kLines;
    for (int c0 = 0; c0 < kLines; c0 += contig ? 4 : kLines)
        for (int j = warp * wj + lj; j < h.cols; j += nw * wj) {
            const int c = c0 + ll;
            double e = 0.0, o = 0.0;
            if (c < nl && j <= half) {
                const double *p = in + base + c * ls;
                const double x = p[j * js];
                if (j == 0 || 2 * j == n) {
                    e = x;
                } else {
                    const double y = p[(n - j) * js];
                    e = x + y;
                    o = x - y;
                }
            }
            E[j * kPitch + c] = e;
            O[j * kPitch + c] = o;
        }
    __syncthreads();
    double cC[U][LT][2], cS[U][LT][2];
    products<U, LT>(h, E, O, cC, cS, warp, nw, lane);
    // this thread's rows k = 8 m + lane / 4 and lines t * 8 + 2 (lane % 4) + {0, 1}
    const int kr = lane >> 2, lc = (lane & 3) * 2;
    if (MODE == kHartleyPoisson) {
        __syncthreads();  // every warp has read e and o
        const double inv_total = 1.0 / ((double)n * (double)a.s);
#pragma unroll
        for (int t = 0; t < LT; ++t)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = t * 8 + lc + q;
                const long tt = min(t0 + c, a.s - 1);
                const int ky = (int)(tt / a.nz), kz = (int)(tt - (long)ky * a.nz);
                const double cz = __ldg(a.cos_z + kz), cy = __ldg(a.cos_y + ky);
                auto scale = [&](double v, int k) {
                    const double lam = 6.0 - 2.0 * cz - 2.0 * __ldg(a.cos_x + k) - 2.0 * cy;
                    return fabs(lam) > 1e-10 ? -v / lam * inv_total : 0.0;
                };
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = (warp + nw * u) * 8 + kr;
                    if (warp + nw * u >= h.tiles || k > half) continue;
                    const double C = cC[u][t][q], S = cS[u][t][q];
                    double e = scale(C + S, k), o = 0.0;
                    if (k != 0 && 2 * k != n) {
                        const double y = scale(C - S, n - k);
                        o = e - y;
                        e = e + y;
                    }
                    E[k * kPitch + c] = e;
                    O[k * kPitch + c] = o;
                }
            }
        __syncthreads();
        products<U, LT>(h, E, O, cC, cS, warp, nw, lane);
    }
    const double sc = MODE == kHartleyScaled ? a.out_scale[comp] : 1.0;
    const double of = MODE == kHartleyScaled ? a.sums[comp] / a.count : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = (warp + nw * u) * 8 + kr;
        if (warp + nw * u >= h.tiles || k > half) continue;
        const bool pair = k != 0 && 2 * k != n;
#pragma unroll
        for (int t = 0; t < LT; ++t)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = t * 8 + lc + q;
                if (c >= nl) continue;
                double *p = out + base + c * ls;
                double x = cC[u][t][q] + cS[u][t][q], y = cC[u][t][q] - cS[u][t][q];
                if (MODE == kHartleyScaled) x = x * sc + of, y = y * sc + of;
                p[k * js] = x;
                if (pair) p[(n - k) * js] = y;
            }
    }
}

long line_tiles(const HartleyArgs &a, int lines) {
    return a.s == 1 ? (a.outer + lines - 1) / lines : a.outer * ((a.s + lines - 1) / lines);
}

template <int U, int MODE, int LT, int W, int CTAS>
void launch_l(const HArgs &h, int ncomp, cudaStream_t s) {
    const size_t smem = (size_t)2 * h.cols * kPitchH<LT> * sizeof(double);
    BINDER_CUDA(cudaFuncSetAttribute(hartley_kernel<U, MODE, LT, W, CTAS>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long gx = line_tiles(h.a, kLinesH<LT>);
    BINDER_CHECK(gx < (1L << 31), "transform grid too large");
    count_launch(), hartley_kernel<U, MODE, LT, W, CTAS>
        <<<dim3((unsigned)gx, (unsigned)ncomp), 32 * ((h.tiles + U - 1) / U), smem, s>>>(h);
    BINDER_CUDA(cudaGetLastError());
}

// 8 lines and a tile per warp where CTAs of 32 lines would be fewer than SMs
template <int MODE>
void launch_mode_h(const HArgs &h, int ncomp, cudaStream_t s) {
    int dev = 0, sms = 148;
    BINDER_CUDA(cudaGetDevice(&dev));
    BINDER_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (line_tiles(h.a, kLinesH<4>) * ncomp < sms) launch_l<1, MODE, 1, 17, 1>(h, ncomp, s);
    else if (h.tiles <= 12) launch_l<2, MODE, 4, 6, 3>(h, ncomp, s);
    else launch_l<2, MODE, 4, 9, 2>(h, ncomp, s);
}

}  // namespace

void HartleyMatrix::init(int n_, cudaStream_t s) {
    release(s);  // of an earlier attempt, whose next allocation failed
    n = n_;
    rows = (n / 2 + 1 + 7) / 8 * 8;
    cols = (n / 2 + 1 + 3) / 4 * 4;
    std::vector<double> host((size_t)2 * rows * cols, 0.0);
    const double pi = 3.14159265358979323846;
    // n angles serve all the entries (a cosine and a sine per entry took 0.7 ms for the three
    // axes of a 160 x 192 x 160 grid)
    std::vector<double> ct(n), st(n);
    for (int m = 0; m < n; ++m) {
        const double ang = 2.0 * pi * (double)m / n;
        ct[m] = std::cos(ang);
        st[m] = std::sin(ang);
    }
    for (int k = 0; k <= n / 2; ++k)
        for (int j = 0, m = 0; j <= n / 2; ++j) {
            host[(size_t)k * cols + j] = ct[m];  // m = j k mod n
            host[(size_t)(rows + k) * cols + j] = st[m];
            m += k;
            if (m >= n) m -= n;
        }
    dev = dev_alloc_n<double>(host.size(), s);
    BINDER_CUDA(cudaMemcpyAsync(dev, host.data(), host.size() * sizeof(double),
                                cudaMemcpyHostToDevice, s));
    BINDER_CUDA(cudaStreamSynchronize(s));  // `host` goes out of scope
}

void HartleyMatrix::release(cudaStream_t s) { dev_free_p(dev, s); }

void launch_hartley(const HartleyArgs &a, const HartleyMatrix &H, HartleyMode mode, int ncomp,
                    cudaStream_t s) {
    BINDER_CHECK(H.n >= 1 && H.n <= 256, "transform axis length must be in [1, 256]");
    BINDER_CHECK(mode != kHartleyPoisson || a.outer == 1,
                 "the Poisson scaling runs on the outermost axis");
    HArgs h{};
    h.a = a;
    h.cs = H.dev;
    h.sn = H.dev + (size_t)H.rows * H.cols;
    h.n = H.n;
    h.cols = H.cols;
    h.tiles = H.rows / 8;
    switch (mode) {
        case kHartleyPlain: launch_mode_h<kHartleyPlain>(h, ncomp, s); break;
        case kHartleyScaled: launch_mode_h<kHartleyScaled>(h, ncomp, s); break;
        case kHartleyPoisson: launch_mode_h<kHartleyPoisson>(h, ncomp, s); break;
    }
}

}  // namespace binder
