// Post-processing on the GPU, on a velocity field in the vel_print layout
// [nx][ny][zd][3] held in device memory (the moments of the running state, or
// a vel file uploaded by the caller): the quadrant analysis of the
// reference's quadrant-analysis/src/qUADrantA.c and the two-point
// correlations of its 2pt-correlations program (below).
//
// A field's cells lie one after another, each with its zd * 3 values together,
// so every kernel here takes groups of neighbouring (plane, component) values
// of a cell -- whole sectors of memory -- and runs over the cells.  All sums
// are FP64 in a fixed order (a block's own range of cells or lines first, then
// the blocks' partial sums in block order), so a result does not depend on
// the run; it differs from the reference's sequential sums by rounding only.
//
// Quadrants.  Per wall-normal fluid plane k = 1 .. zd-2: the plane means of u,
// v, w over (x, y); the fluctuations u' = u - <u>, w' = w - <w>; the products
// u'w' summed over the plane and over each quadrant Q1 (u' > 0, w' > 0),
// Q2 (u' < 0, w' > 0), Q3 (u' < 0, w' < 0), Q4 (u' > 0, w' < 0), with the cell
// count of each quadrant (a zero u' or w' falls in none, as in the reference).
#include <cuda_runtime.h>

#include <algorithm>

#include "step_common.cuh"

namespace dnslbm {

constexpr int kQuadThreads = 256;

// Blocks of the kernels that run over all cells: each takes a contiguous
// range, about four blocks per SM's worth.
constexpr int kCellBlocks = 592;
static int cell_blocks(size_t cells) { return (int)std::min<size_t>(kCellBlocks, cells); }

// part[block][zd * 3] sums of the block's cells, one thread per value
__global__ void __launch_bounds__(kQuadThreads) vel_sums_kernel(const double *__restrict__ vel, size_t cells, int zd,
                                                                double *part)
{
    const size_t c0 = cells * blockIdx.x / gridDim.x, c1 = cells * (blockIdx.x + 1) / gridDim.x;
    const int nv = zd * 3;
    for (int e = threadIdx.x; e < nv; e += blockDim.x) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        size_t c = c0;
        for (; c + 4 <= c1; c += 4)
#pragma unroll
            for (int q = 0; q < 4; ++q) s[q] += vel[(c + q) * nv + e];
        for (; c < c1; ++c) s[0] += vel[c * nv + e];
        part[(size_t)blockIdx.x * nv + e] = (s[0] + s[1]) + (s[2] + s[3]);
    }
}

// out[e] = scale * sum over the blocks of part[block][e]; one warp per value
__global__ void column_sum_kernel(const double *__restrict__ part, int nblocks, int nv, double scale, double *out)
{
    const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= nv) return;
    double s[1] = {0.0};
    for (int b = lane; b < nblocks; b += 32) s[0] += part[(size_t)b * nv + e];
    warp_sum<1>(s);
    if (lane == 0) out[e] = scale * s[0];
}

// mean[zd][3]: plane means; part holds cell_blocks * zd * 3 doubles
static void plane_means(const double *vel, int nx, int ny, int zd, double *part, double *mean, cudaStream_t s)
{
    const size_t cells = (size_t)nx * ny;
    const int nb = cell_blocks(cells);
    vel_sums_kernel<<<nb, kQuadThreads, 0, s>>>(vel, cells, zd, part);
    column_sum_kernel<<<(zd * 3 + 7) / 8, 256, 0, s>>>(part, nb, zd * 3, 1.0 / (double)cells, mean);
}

// part[block][zd][9] of the block's cells: 0..3 u'w' summed per quadrant,
// 4..7 the quadrants' cell counts, 8 u'w' summed; one thread per plane
__global__ void __launch_bounds__(kQuadThreads) quadrant_kernel(const double *__restrict__ vel,
                                                                const double *__restrict__ mean, size_t cells, int zd,
                                                                double *part)
{
    const size_t c0 = cells * blockIdx.x / gridDim.x, c1 = cells * (blockIdx.x + 1) / gridDim.x;
    for (int k = threadIdx.x; k < zd; k += blockDim.x) {
        const double mu = mean[k * 3 + 0], mw = mean[k * 3 + 2];
        double s[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) s[i] = 0.0;
#pragma unroll 4
        for (size_t c = c0; c < c1; ++c) {
            const double *v = vel + (c * zd + k) * 3;
            const double up = v[0] - mu, wp = v[2] - mw, p = up * wp;
            s[8] += p;
            const int q = up > 0.0 ? (wp > 0.0 ? 0 : (wp < 0.0 ? 3 : -1)) : (up < 0.0 ? (wp > 0.0 ? 1 : (wp < 0.0 ? 2 : -1)) : -1);
#pragma unroll
            for (int a = 0; a < 4; ++a)
                if (q == a) s[a] += p, s[4 + a] += 1.0;
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) part[((size_t)blockIdx.x * zd + k) * 9 + i] = s[i];
    }
}

// Scratch of launch_quadrant, in doubles.
size_t quadrant_scratch(int nx, int ny, int zd) { return (size_t)cell_blocks((size_t)nx * ny) * zd * 9; }

// mean [zd][3] and out [zd][9] in device memory
void launch_quadrant(const double *vel, int nx, int ny, int zd, double *scratch, double *mean, double *out, cudaStream_t s)
{
    const size_t cells = (size_t)nx * ny;
    const int nb = cell_blocks(cells);
    plane_means(vel, nx, ny, zd, scratch, mean, s);
    quadrant_kernel<<<nb, kQuadThreads, 0, s>>>(vel, mean, cells, zd, scratch);
    column_sum_kernel<<<(zd * 9 + 7) / 8, 256, 0, s>>>(scratch, nb, zd * 9, 1.0, out);
}

// ------------------------------------------------------------------ correlations
// Two-point velocity correlations of the reference's 2pt-correlations
// program (mean_subtract.c, xcorrel.c, ycorrel.c), one velocity field:
//   ua[k]              the subtracted mean of plane k: the plane means of
//                      u, v, w over (x, y), made symmetric about the channel
//                      centre (u, v even, w odd: mean_subtract.c:178-196);
//                      0 on the wall planes, which are not shifted;
//   xcorl[k][d][c]     sum over (x, y) of u'_c(x, y, k) u'_c(x + d, y, k),
//                      d = 0 .. nx-1 periodic (xcorrel.c);
//   ycorl[k][d][c]     sum over (x, y) of u'_c(x, y, k) u'_c(x, y + d, k),
//                      d = 0 .. ny-1 periodic (ycorrel.c).
// Both are one kernel: the autocorrelation of every line along x (or y) of
// every (plane, component), summed over the lines.  A periodic
// autocorrelation is even in the lag, so lags 0 .. len/2 are computed.  FP64
// throughout: O(len^2 / 2) multiply-adds per line, which bound the kernel
// (their FP64 rate) as long as operands come from registers: a thread keeps
// eight neighbouring lags and slides a window of eight elements over the
// line, two shared-memory loads per eight multiply-adds (one lag per load
// before: 402x201x130, both directions 13.6 ms).

constexpr int kCorrLags = 8;
constexpr int kCorrMaxLine = 2048;

__global__ void corr_mean_kernel(const double *__restrict__ mean, int zd, double *ua /* [zd][3] */)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= zd) return;
    if (k == 0 || k == zd - 1) {
        ua[k * 3] = ua[k * 3 + 1] = ua[k * 3 + 2] = 0.0;
        return;
    }
    const int kk = zd - 1 - k;
    ua[k * 3 + 0] = 0.5 * (mean[k * 3 + 0] + mean[kk * 3 + 0]);
    ua[k * 3 + 1] = 0.5 * (mean[k * 3 + 1] + mean[kk * 3 + 1]);
    ua[k * 3 + 2] = 0.5 * (mean[k * 3 + 2] - mean[kk * 3 + 2]);
}

// Shape of the line kernel for lines of len elements: kc (plane, component)
// values per block, lg threads (of eight lags each) per value.
struct CorrShape {
    int lg, kc, row;  // row: doubles of one line in shared memory
    size_t smem;
};
static CorrShape corr_shape(int len)
{
    CorrShape c;
    c.lg = (len / 2 + 1 + kCorrLags - 1) / kCorrLags;
    const int last = (len + kCorrLags - 1) / kCorrLags * kCorrLags + kCorrLags * (c.lg + 1);
    c.row = last + last / kCorrLags + 1;
    c.kc = 16;
    while (c.kc > 1 && (c.kc * c.lg > 512 || (size_t)c.kc * c.row * sizeof(double) > 200 * 1024)) c.kc /= 2;
    c.smem = (size_t)c.kc * c.row * sizeof(double);
    return c;
}
// line ranges per (plane, component) group: enough blocks for every SM
static int corr_chunks(int len, int nlines, int zd)
{
    const int groups = (zd * 3 + corr_shape(len).kc - 1) / corr_shape(len).kc;
    return std::max(1, std::min(nlines, (4 * 148 + groups - 1) / groups));
}

// Element i of line m, value e: vel[i * istride + m * mstride + e], minus
// ua[e].  part [chunks][zd * 3][lags], lags = lg * 8.  Shared memory holds the
// block's kc lines, each element at e + e / 8 (the threads of a value start
// eight elements apart: without the padding they would meet in a bank), the
// line's start repeated behind its end.
__global__ void __launch_bounds__(512) line_corr_kernel(const double *__restrict__ vel, const double *__restrict__ ua, int len,
                                                        int nlines, size_t istride, size_t mstride, int nv, int kc, int lg,
                                                        int row, double *part)
{
    extern __shared__ double ln[];
    const int e0 = blockIdx.x * kc, ne = min(kc, nv - e0);
    const int m0 = (int)((long long)nlines * blockIdx.y / gridDim.y), m1 = (int)((long long)nlines * (blockIdx.y + 1) / gridDim.y);
    const int v = threadIdx.x / lg, g = threadIdx.x - v * lg;
    const int last = (len + kCorrLags - 1) / kCorrLags * kCorrLags + kCorrLags * (lg + 1);
    double acc[kCorrLags];
#pragma unroll
    for (int q = 0; q < kCorrLags; ++q) acc[q] = 0.0;
    const double *line = ln + (size_t)v * row;
    for (int m = m0; m < m1; ++m) {
        __syncthreads();  // the previous line is no longer read
        for (int t = threadIdx.x; t < last * kc; t += blockDim.x) {
            const int i = t / kc, q = t - i * kc;
            if (q < ne) ln[(size_t)q * row + i + i / kCorrLags] =
                            vel[(size_t)(i % len) * istride + (size_t)m * mstride + e0 + q] - ua[e0 + q];
        }
        __syncthreads();
        if (v >= ne) continue;
        // window w[(j + q) % 8] holds element i + j + 8 g + q
        double w[kCorrLags];
        const double *base = line + (size_t)g * (kCorrLags + 1);  // element 8 g
#pragma unroll
        for (int q = 0; q < kCorrLags - 1; ++q) w[q] = base[q];
        const int whole = len / kCorrLags;
        for (int b = 0; b < whole; ++b) {
            const double *ai = line + (size_t)b * (kCorrLags + 1), *wi = base + (size_t)b * (kCorrLags + 1);
#pragma unroll
            for (int j = 0; j < kCorrLags; ++j) {
                const int n = j + kCorrLags - 1;
                w[n % kCorrLags] = wi[n + n / kCorrLags];
                const double a = ai[j];
#pragma unroll
                for (int q = 0; q < kCorrLags; ++q) acc[q] = fma(a, w[(j + q) % kCorrLags], acc[q]);
            }
        }
        for (int i = whole * kCorrLags; i < len; ++i) {
            const double a = line[i + i / kCorrLags];
#pragma unroll
            for (int q = 0; q < kCorrLags; ++q) {
                const int n = i + g * kCorrLags + q;
                acc[q] = fma(a, line[n + n / kCorrLags], acc[q]);
            }
        }
    }
    if (v >= ne) return;
    double *out = part + ((size_t)blockIdx.y * nv + e0 + v) * lg * kCorrLags + g * kCorrLags;
#pragma unroll
    for (int q = 0; q < kCorrLags; ++q) out[q] = acc[q];
}

// out [zd][len][3] = sum over the chunks, in chunk order; lag len - d as d
__global__ void corr_reduce_kernel(const double *__restrict__ part, int nchunks, int len, int lags, int zd, double *out)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)zd * 3 * len;
    if (idx >= n) return;
    const int c = (int)(idx % 3);
    const size_t t = idx / 3;
    const int d = (int)(t % len), k = (int)(t / len);
    const int lag = d <= len / 2 ? d : len - d;
    double s = 0.0;
    for (int ch = 0; ch < nchunks; ++ch) s += part[((size_t)ch * zd * 3 + k * 3 + c) * lags + lag];
    out[idx] = s;
}

static size_t corr_part(int len, int nlines, int zd)
{
    return (size_t)corr_chunks(len, nlines, zd) * zd * 3 * corr_shape(len).lg * kCorrLags;
}

// Scratch of launch_correlations, in doubles.
size_t correlation_scratch(int nx, int ny, int zd)
{
    return (size_t)zd * 3 + std::max({(size_t)cell_blocks((size_t)nx * ny) * zd * 3, corr_part(nx, ny, zd), corr_part(ny, nx, zd)});
}

int correlation_max_line() { return kCorrMaxLine; }

// vel in device memory; scratch of correlation_scratch doubles; xcorl
// [zd][nx][3], ycorl [zd][ny][3], ua [zd][3] in device memory.
cudaError_t launch_correlations(const double *vel, int nx, int ny, int zd, double *scratch, double *xcorl, double *ycorl,
                                double *ua, cudaStream_t s)
{
    if (nx > correlation_max_line() || ny > correlation_max_line()) return cudaErrorInvalidValue;
    double *mean = scratch, *part = scratch + (size_t)zd * 3;
    plane_means(vel, nx, ny, zd, part, mean, s);
    corr_mean_kernel<<<(zd + 127) / 128, 128, 0, s>>>(mean, zd, ua);
    const int nv = zd * 3;
    for (int dir = 0; dir < 2; ++dir) {
        const int len = dir ? ny : nx, nlines = dir ? nx : ny;
        const size_t sx = (size_t)ny * nv, sy = nv;
        const CorrShape c = corr_shape(len);
        const int chunks = corr_chunks(len, nlines, zd);
        cudaError_t e = cudaFuncSetAttribute(line_corr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
        if (e != cudaSuccess) return e;
        line_corr_kernel<<<dim3((nv + c.kc - 1) / c.kc, chunks), c.kc * c.lg, c.smem, s>>>(
            vel, ua, len, nlines, dir ? sy : sx, dir ? sx : sy, nv, c.kc, c.lg, c.row, part);
        corr_reduce_kernel<<<(unsigned)(((size_t)nv * len + 255) / 256), 256, 0, s>>>(part, chunks, len, c.lg * kCorrLags, zd,
                                                                                    dir ? ycorl : xcorl);
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------------ spectra
// One-dimensional energy spectra of the reference's e-spectra program
// (e-spectra/src/1d-spectra.c), one velocity field.  Per fluid plane k and
// component c: the 2-D real-to-complex DFT over (x, y) (FFTW's r2c_2d,
// C[i][j] = sum_{x,y} u(x, y) e^{-2 pi i (i x / nx + j y / ny)}, i < nx,
// j <= ny/2), scaled by 2 / (2 nx ny) (:131-143), the (0, 0) mode set to 0
// (:146-151), then p = 0.5 fac_j |C|^2 with fac_0 = 1, fac_j = 2 otherwise
// (:156-172), summed over j into E_x[i][k] and over i into E_y[j][k]; the
// wall planes are 0.
//
// The DFT is evaluated directly in FP64 for any length (two passes: the half
// spectrum along y of every x line, then the transform along x of every kept
// y mode), with exact twiddle factors sincospi(2 m / n), m = n * index mod n.
// Elements x and n - x enter with the same cosine and opposite sines, so each
// pass works on their sums and differences: half the terms along y, and along
// x half the terms and half the modes (mode n - i from the same sums as i).
// FP64 multiply-adds bound both passes; a thread takes one mode of many
// (plane, component) values at once, so that one twiddle look-up serves them
// all and their elements are broadcast loads (one value per thread before:
// 402x201x128 FP64 field 19.6 ms).
// The first pass leaves V[x][group][j][kKcY] complex, a group being kKcY
// neighbouring (plane, component) values: both passes move it in whole lines.

constexpr int kKcY = 16;  // values per group

// twiddles: tw[m] = (cos(2 pi m / n), sin(2 pi m / n)), m < n
__global__ void spec_twiddle_kernel(int n, double2 *tw)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    double s, c;
    sincospi(2.0 * (double)m / (double)n, &s, &c);
    tw[m] = make_double2(c, s);
}

// grid (groups * (kKcY / KC), nx): the KC values of one line x
template <int KC>
__global__ void __launch_bounds__(128) spec_y_kernel(const double *__restrict__ vel, const double2 *__restrict__ twy, int nx,
                                                     int ny, int zd, int nj, double2 *V)
{
    extern __shared__ double sm[];
    const int nh = ny / 2 + 1;  // terms after folding
    double2 *tw = reinterpret_cast<double2 *>(sm);
    double *ev = sm + 2 * ny, *od = ev + (size_t)nh * KC;
    const int x = blockIdx.y, e0 = blockIdx.x * KC, nv = (zd - 2) * 3;
    const double *src = vel + ((size_t)x * ny * zd + 1) * 3 + e0;  // plane 1 on
    for (int m = threadIdx.x; m < ny; m += blockDim.x) tw[m] = twy[m];
    for (int t = threadIdx.x; t < nh * KC; t += blockDim.x) {
        const int y = t / KC, q = t - y * KC, yy = ny - y;
        const double a = e0 + q < nv ? src[(size_t)y * zd * 3 + q] : 0.0;
        const bool pair = y != 0 && yy != y;
        const double b = pair && e0 + q < nv ? src[(size_t)yy * zd * 3 + q] : 0.0;
        ev[t] = a + b;
        od[t] = pair ? a - b : 0.0;
    }
    __syncthreads();
    const int g = e0 / kKcY, q0 = e0 % kKcY, groups = (nv + kKcY - 1) / kKcY;
    for (int j = threadIdx.x; j < nj; j += blockDim.x) {
        double re[KC], im[KC];
#pragma unroll
        for (int q = 0; q < KC; ++q) re[q] = im[q] = 0.0;
        int m = 0;
        for (int y = 0; y < nh; ++y) {
            const double2 w = tw[m];
            const double *e = ev + (size_t)y * KC, *o = od + (size_t)y * KC;
#pragma unroll
            for (int q = 0; q < KC; ++q) {
                re[q] = fma(e[q], w.x, re[q]);
                im[q] = fma(o[q], -w.y, im[q]);
            }
            m += j;
            if (m >= ny) m -= ny;
        }
        double2 *out = V + (((size_t)x * groups + g) * nj + j) * kKcY + q0;
#pragma unroll
        for (int q = 0; q < KC; ++q) out[q] = make_double2(re[q], im[q]);
    }
}

// grid (groups * (kKcY / KC), chunks): KC values of the modes j of the
// chunk.  ey [nzf * 3][nj]; part[chunk][nzf * 3][nx].
template <int KC, bool TWS>
__global__ void __launch_bounds__(256) spec_x_kernel(const double2 *__restrict__ V, const double2 *__restrict__ twx, int nx,
                                                     int nj, int nv, int jb, double scale, double *ey, double *part)
{
    extern __shared__ double sm[];
    __shared__ double red[32 * KC];
    const int nh = nx / 2 + 1;
    double4 *eo = reinterpret_cast<double4 *>(sm);  // [nh][KC]: sum (re, im), difference (re, im)
    double2 *tws = reinterpret_cast<double2 *>(eo + (size_t)nh * KC);
    const int e0 = blockIdx.x * KC, g = e0 / kKcY, q0 = e0 % kKcY, groups = (nv + kKcY - 1) / kKcY;
    if (TWS)
        for (int m = threadIdx.x; m < nx; m += blockDim.x) tws[m] = twx[m];
    const double2 *tw = TWS ? tws : twx;
    const int j0 = blockIdx.y * jb, j1 = min(j0 + jb, nj);
    double *pout = part + ((size_t)blockIdx.y * nv + e0) * nx;
    for (int j = j0; j < j1; ++j) {
        __syncthreads();
        for (int t = threadIdx.x; t < nh * KC; t += blockDim.x) {
            const int x = t / KC, q = t - x * KC, xx = nx - x;
            const double2 a = V[(((size_t)x * groups + g) * nj + j) * kKcY + q0 + q];
            const bool pair = x != 0 && xx != x;
            const double2 b = pair ? V[(((size_t)xx * groups + g) * nj + j) * kKcY + q0 + q] : make_double2(0.0, 0.0);
            eo[t] = pair ? double4{a.x + b.x, a.y + b.y, a.x - b.x, a.y - b.y} : double4{a.x, a.y, 0.0, 0.0};
        }
        __syncthreads();
        const double fac = j == 0 ? 0.5 : 1.0;
        double sy[KC];
#pragma unroll
        for (int q = 0; q < KC; ++q) sy[q] = 0.0;
        for (int i = threadIdx.x; i < nh; i += blockDim.x) {
            double pr[KC], pi[KC], rr[KC], ri[KC];
#pragma unroll
            for (int q = 0; q < KC; ++q) pr[q] = pi[q] = rr[q] = ri[q] = 0.0;
            int m = 0;
            for (int x = 0; x < nh; ++x) {
                const double2 w = tw[m];
                const double4 *v = eo + (size_t)x * KC;
#pragma unroll
                for (int q = 0; q < KC; ++q) {
                    const double4 u = v[q];
                    pr[q] = fma(u.x, w.x, pr[q]);
                    pi[q] = fma(u.y, w.x, pi[q]);
                    rr[q] = fma(u.z, w.y, rr[q]);
                    ri[q] = fma(u.w, w.y, ri[q]);
                }
                m += i;
                if (m >= nx) m -= nx;
            }
            // C[i] = P - i R, C[nx - i] = P + i R
            const bool two = i != 0 && 2 * i != nx;
#pragma unroll
            for (int q = 0; q < KC; ++q) {
                if (e0 + q >= nv) continue;
                const double ar = scale * (pr[q] + ri[q]), ai = scale * (pi[q] - rr[q]);
                const double br = scale * (pr[q] - ri[q]), bi = scale * (pi[q] + rr[q]);
                const double pa = i == 0 && j == 0 ? 0.0 : fac * (ar * ar + ai * ai), pb = fac * (br * br + bi * bi);
                double *o = pout + (size_t)q * nx;
                o[i] = (j == j0 ? 0.0 : o[i]) + pa;
                if (two) o[nx - i] = (j == j0 ? 0.0 : o[nx - i]) + pb;
                sy[q] += two ? pa + pb : pa;
            }
        }
        block_sum<KC>(sy, red);  // over i, in a fixed order
        if (threadIdx.x == 0)
#pragma unroll
            for (int q = 0; q < KC; ++q)
                if (e0 + q < nv) ey[(size_t)(e0 + q) * nj + j] = sy[q];
    }
}

// E_x[k][c][i] = sum over the j chunks of part, in chunk order
__global__ void spec_reduce_kernel(const double *__restrict__ part, int nchunks, int nx, int nzf, double *ex)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)nzf * 3 * nx;
    if (idx >= n) return;
    double s = 0.0;
    for (int ch = 0; ch < nchunks; ++ch) s += part[(size_t)ch * n + idx];
    ex[idx] = s;
}

static int spec_chunk(int nj) { return std::max(1, std::min(8, (nj + 11) / 12)); }

// Scratch of launch_spectra, in doubles.
size_t spectra_scratch(int nx, int ny, int zd)
{
    const int nj = ny / 2 + 1, nv = (zd - 2) * 3, groups = (nv + kKcY - 1) / kKcY, jb = spec_chunk(nj);
    return 2 * (size_t)(nx + ny) + 2 * (size_t)nx * groups * nj * kKcY + (size_t)((nj + jb - 1) / jb) * nv * nx;
}

template <int KC>
static cudaError_t launch_spec_y(const double *vel, const double2 *twy, int nx, int ny, int zd, int nj, double2 *V, size_t smem,
                                 cudaStream_t s)
{
    const int nv = (zd - 2) * 3, groups = (nv + kKcY - 1) / kKcY;
    const cudaError_t e = cudaFuncSetAttribute(spec_y_kernel<KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int threads = std::min(128, (nj + 31) / 32 * 32);
    for (int x0 = 0; x0 < nx; x0 += 65535) {  // one grid row per x
        const int n = std::min(65535, nx - x0);
        spec_y_kernel<KC><<<dim3(groups * (kKcY / KC), n), threads, smem, s>>>(
            vel + (size_t)x0 * ny * zd * 3, twy, nx, ny, zd, nj, V + (size_t)x0 * groups * nj * kKcY);
    }
    return cudaGetLastError();
}

template <int KC, bool TWS>
static cudaError_t launch_spec_x(const double2 *V, const double2 *twx, int nx, int nj, int nv, int jb, double scale, double *ey,
                                 double *part, size_t smem, cudaStream_t s)
{
    const int groups = (nv + kKcY - 1) / kKcY;
    const cudaError_t e = cudaFuncSetAttribute(spec_x_kernel<KC, TWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int threads = std::min(256, (nx / 2 + 1 + 31) / 32 * 32);
    spec_x_kernel<KC, TWS><<<dim3(groups * (kKcY / KC), (nj + jb - 1) / jb), threads, smem, s>>>(V, twx, nx, nj, nv, jb, scale,
                                                                                              ey, part);
    return cudaGetLastError();
}

// ex [zd-2][3][nx], ey [zd-2][3][ny/2+1] in device memory (fluid planes).
// Values per block: as many as shared memory holds for the line length.
cudaError_t launch_spectra(const double *vel, int nx, int ny, int zd, double *scratch, double *ex, double *ey, cudaStream_t s)
{
    const int nj = ny / 2 + 1, nzf = zd - 2, nv = nzf * 3, groups = (nv + kKcY - 1) / kKcY, jb = spec_chunk(nj);
    const int chunks = (nj + jb - 1) / jb;
    double2 *twx = reinterpret_cast<double2 *>(scratch), *twy = twx + nx;
    double2 *V = twy + ny;
    double *part = reinterpret_cast<double *>(V + (size_t)nx * groups * nj * kKcY);
    const size_t cap = 220 * 1024;
    auto smem_y = [&](int kc) { return (2 * (size_t)ny + 2 * (size_t)(ny / 2 + 1) * kc) * sizeof(double); };
    auto smem_x = [&](int kc, bool tws) { return ((size_t)(nx / 2 + 1) * kc * 4 + (tws ? 2 * (size_t)nx : 0)) * sizeof(double); };
    spec_twiddle_kernel<<<(nx + 255) / 256, 256, 0, s>>>(nx, twx);
    spec_twiddle_kernel<<<(ny + 255) / 256, 256, 0, s>>>(ny, twy);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (smem_y(16) <= cap) e = launch_spec_y<16>(vel, twy, nx, ny, zd, nj, V, smem_y(16), s);
    else if (smem_y(4) <= cap) e = launch_spec_y<4>(vel, twy, nx, ny, zd, nj, V, smem_y(4), s);
    else e = launch_spec_y<1>(vel, twy, nx, ny, zd, nj, V, smem_y(1), s);
    if (e != cudaSuccess) return e;
    const double scale = 2.0 * (1.0 / (2.0 * nx * ny));
    if (smem_x(8, true) <= cap) e = launch_spec_x<8, true>(V, twx, nx, nj, nv, jb, scale, ey, part, smem_x(8, true), s);
    else if (smem_x(2, true) <= cap) e = launch_spec_x<2, true>(V, twx, nx, nj, nv, jb, scale, ey, part, smem_x(2, true), s);
    else e = launch_spec_x<1, false>(V, twx, nx, nj, nv, jb, scale, ey, part, smem_x(1, false), s);
    if (e != cudaSuccess) return e;
    spec_reduce_kernel<<<(unsigned)(((size_t)nv * nx + 255) / 256), 256, 0, s>>>(part, chunks, nx, nzf, ex);
    return cudaGetLastError();
}

}  // namespace dnslbm
