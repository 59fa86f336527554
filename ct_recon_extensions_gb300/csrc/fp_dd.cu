// Distance-driven parallel forward projection and the reference's
// distance-driven gradient (src/fp_par_2d.cc:396-653).
//
// Forward: a ray's footprint on each line of the marched axis is [left,
// right] (running FP64 sums from the channel's centre +- half width).  It
// averages the trapezoid (p[i] + p[i+1]) / 2 of neighbouring pixels over the
// pixel intervals [i, i+1] it covers, weighted by the covered length, and the
// line adds tsum / lsum.  The reference's pixel loop runs an unsigned index
// from floor(left): a negative floor converts (undefined in C++) to a huge
// value on the x86-64 build that its fixtures come from, so such a line adds
// nothing; intervals from nx-1 on are skipped.  Positions, the line's
// interval range and the two partial lengths (first and last interval) are
// FP64 as in the reference, so every decision is the reference's; for
// T = float the sums run in FP32 as the reference's T sums do.  One thread per
// ray.
//
// Grad (the reference's, not the adjoint of the normalised forward): per
// pixel and view the channel footprint around the pixel's channel mid (mid -
// offset .. mid + offset, one-sided at the image edges) gathers
// length * proj / 2 over channels ceil(left - 0.5) .. floor(right + 0.5); a
// negative first channel skips the view (the same unsigned index), and
// channels past ns read on into the next view's row as the reference's
// unchecked index does (0 past the last view).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "ctr_common.cuh"
#include "dd_window.h"
#include "fp_setup.cuh"

namespace ctr {
namespace {

constexpr int kDdThreads = 128;
constexpr double kDdPi = 3.14159265358979323846;

// Fraction of a 32.32 fixed-point value, from its low word's top 23 bits.
__device__ __forceinline__ float dd_frac(long long X)
{
    return __uint_as_float(0x3F800000u | (static_cast<unsigned>(X) >> 9)) - 1.0f;
}

// Copies of the image with its lines as rows (rows: image rows, cols: image
// columns), each row padded with kDdPad zeros; 32 x 32 tiles.
constexpr int kDdPad = 3;
__global__ void __launch_bounds__(256)
    dd_copies(const float* __restrict__ img, float* __restrict__ rows, float* __restrict__ cols, int n)
{
    __shared__ float t[32][33];
    const size_t off = static_cast<size_t>(blockIdx.z) * n * n, w = n + kDdPad, poff = blockIdx.z * n * w;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int x = x0 + tx, y = y0 + r;
        const float v = x < n && y < n ? img[off + static_cast<size_t>(y) * n + x] : 0.0f;
        t[r][tx] = v;
        if (x < w && y < n) rows[poff + y * w + x] = v;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8)
        if (x0 + r < n && y0 + tx < w) cols[poff + (x0 + r) * w + y0 + tx] = t[tx][r];
}

// One ray of the forward with the reference's own arithmetic: FP64 edges,
// interval range and lengths; sums in T (FP32 for T = float).
template <typename T>
__device__ T dd_ray_exact(const T* __restrict__ I, const double* __restrict__ b, int ux, int nl, int nal,
                          int nx)
{
    const size_t step_line = ux ? static_cast<size_t>(nx) : 1;   // next line
    const size_t step_pix = ux ? 1 : static_cast<size_t>(nx);    // next pixel along the line
    const double off = b[1];
    double left = __dsub_rn(b[0], b[2]), right = __dadd_rn(b[0], b[2]);
    if (left > right) {
        const double t = left;
        left = right;
        right = t;
    }
    T sum = 0;
    for (int l = 0; l < nl; ++l) {
        const double fl = floor(left), cr = ceil(right);
        T tsum = 0, lsum = 0;
        if (fl >= 0.0) {
            // intervals i0 .. (i < cr), all but those from nal - 1 on
            const int i0 = static_cast<int>(fl);
            const int iend = cr < static_cast<double>(nal - 1) ? static_cast<int>(cr) : nal - 1;
            const T* line = I + static_cast<size_t>(l) * step_line;
            for (int i = i0; i < iend; ++i) {
                const double a = static_cast<double>(i + 1) < right ? static_cast<double>(i + 1) : right;
                const double c = static_cast<double>(i) > left ? static_cast<double>(i) : left;
                const double len = a - c;
                const T p0 = line[static_cast<size_t>(i) * step_pix];
                const T p1 = line[static_cast<size_t>(i + 1) * step_pix];
                if constexpr (sizeof(T) == 4) {
                    const float lf = static_cast<float>(len);
                    tsum = fmaf(lf, (p0 + p1) * 0.5f, tsum);
                    lsum += lf;
                } else {
                    tsum += len * (p0 + p1) / 2;
                    lsum += len;
                }
            }
        }
        if (lsum > 0) sum += tsum / lsum;
        left += off;
        right += off;
    }
    return sum;
}

// The reference's loop, one thread per ray: FP64, and FP32 where there is no room
// for an image's copies.
template <typename T>
__global__ void __launch_bounds__(kDdThreads)
    fp_dd_rays(const T* __restrict__ img, T* __restrict__ proj, const double* __restrict__ sincos,
               const double* __restrict__ bo, const int* __restrict__ usex, int ns, int na, int nx, int ny,
               double dx, double dy, size_t img_stride, size_t proj_stride)
{
    const long long ray = static_cast<long long>(blockIdx.x) * kDdThreads + threadIdx.x;
    if (ray >= static_cast<long long>(na) * ns) return;
    const int ia = static_cast<int>(ray / ns);
    const int ux = usex[ia];
    const T w = static_cast<T>(ux ? fabs(dy / sincos[2 * ia + 1]) : fabs(dx / sincos[2 * ia]));
    const T sum = dd_ray_exact<T>(img + blockIdx.y * img_stride, bo + 3 * ray, ux, ux ? ny : nx, ux ? nx : ny, nx);
    proj[blockIdx.y * proj_stride + ray] = sum * w;
}

// FP32 forward.  The reference's discontinuous decisions come down to which
// lines count: a line adds tsum / lsum iff its footprint start satisfies
// 0 <= left < n-1 (a negative start skips it; from n-1 on no interval is
// left), a contiguous range of lines since left is a running sum.  That range
// is decided as the reference decides it (axis_range, and a line exactly at
// n-1 dropped after an exact check).  Inside it both edges march in 32.32
// fixed point, and the covered lengths are FP32 relative to the first
// interval; everything else varies continuously with the edges.  Lines of
// column-marching views read the transposed copy.  Rays outside the
// fixed-point range take dd_ray_exact.
//
// A footprint's width is the same on every line, and up to two pixels (every
// view when ds <= sqrt(2) dx) it covers at most three intervals: all lines but
// those at the image's edges run a loop without an interval count or a
// division, its sums scaled by the common width's reciprocal four lines at a time
// (one sum over all lines cost digits: noise on 512^2 5.3e-7 from FP64, now 2.2e-7,
// 3.8e-7 line by line with a division each).  One lane per ray, a
// block's lanes on adjacent channels of one view, the warp's rays on the same
// line, so that each load reads adjacent pixels.  Blocks follow one another by
// view, chunk of channels by chunk: neighbouring views' rays through the same
// lines, and the short rays of the detector's first eighth for the last blocks (calls of 512^2 x
// 720 x 729 with a quarter channel's offset: 284 us view by view, 260 so, three
// images 703 and 667; without the offset 278 either way; from the middle outwards,
// as in the ray casting, 320).  Issue bound.
constexpr int kDdRayThreads = 64, kDdUnroll = 4;

// A counted line's tsum / lsum, with the edges' clamps.
__device__ __forceinline__ float dd_line(const float* __restrict__ line, long long xl, long long xr, int n)
{
    const int h = static_cast<int>(xl >> 32);
    const int i0 = min(max(h, 0), n - 2);
    // the start relative to interval i0 (clamped: the fixed-point start may
    // sit a hair outside [0, n-1) where the exact one is inside)
    const float lr = h == i0 ? dd_frac(xl) : (h < 0 ? 0.0f : 1.0f);
    const int hr = static_cast<int>(xr >> 32);
    const float rr = static_cast<float>(hr - i0) + dd_frac(xr);
    const int ie = min(hr + (static_cast<unsigned>(xr) != 0u ? 1 : 0), n - 1);
    float tsum = 0.0f, lsum = 0.0f;
    for (int i = i0; i < ie; ++i) {
        const float j = static_cast<float>(i - i0);
        const float len = fmaxf(fminf(j + 1.0f, rr) - fmaxf(j, lr), 0.0f);
        tsum = fmaf(len, (__ldg(line + i) + __ldg(line + i + 1)) * 0.5f, tsum);
        lsum += len;
    }
    // a counted line always covers part of interval i0; where the clamped
    // fixed-point edges leave no length, that sliver's trapezoid is the mean
    return lsum > 0.0f ? tsum / lsum : (__ldg(line + i0) + __ldg(line + i0 + 1)) * 0.5f;
}

__global__ void __launch_bounds__(kDdRayThreads, 14)
    fp_dd_f32(const float* __restrict__ img, const float* __restrict__ rows, const float* __restrict__ cols,
              float* __restrict__ proj,
              const double* __restrict__ sincos, const double* __restrict__ bo, const int* __restrict__ usex,
              int ns, unsigned chunks, int n, double dx, double dy, size_t img_stride, size_t proj_stride)
{
    // each chunk of channels for every view, from an eighth of the detector on
    const unsigned na = gridDim.x / chunks, rank = blockIdx.x / na, ia = blockIdx.x - rank * na;
    const unsigned chunk = rank + chunks / 8 < chunks ? rank + chunks / 8 : rank + chunks / 8 - chunks;
    const int is = static_cast<int>(chunk * kDdRayThreads + threadIdx.x);
    const size_t ray = static_cast<size_t>(ia) * ns + is;
    const int ux = usex[ia];
    const size_t w = n + kDdPad;
    const float* I = (ux ? rows : cols) + blockIdx.y * n * w;  // lines are rows of I
    long long xl = 0, xr = 0, S = 0;
    int k0 = 1, k1 = 0;  // the lines left to the loop
    float sum = 0.0f;
    if (is < ns) {
        const double* b = bo + 3 * ray;
        const double off = b[1];
        double left0 = __dsub_rn(b[0], b[2]), right0 = __dadd_rn(b[0], b[2]);
        if (left0 > right0) {
            const double t = left0;
            left0 = right0;
            right0 = t;
        }
        const int er = static_cast<int>((double_bits(right0) >> 52) & 0x7FF);
        const int el = static_cast<int>((double_bits(left0) >> 52) & 0x7FF);
        const int eo = static_cast<int>((double_bits(off) >> 52) & 0x7FF);
        if (er >= 1043 || el >= 1043 || eo >= 1025 || n < 2) {  // beyond the fixed-point range
            sum = dd_ray_exact<float>(img + blockIdx.y * img_stride, b, ux, n, n, n);
        } else {
            long long XL;
            axis_range(left0, off, n, n, &XL, &S, &k0, &k1);
            // a start exactly at n-1 leaves no interval: the range's end there drops
            if (k0 <= k1) {
                const double lim = static_cast<double>(n - 1);
                const long long L = static_cast<long long>(n - 1) << 32, T = tie_units(n);
                if (off == 0.0) {
                    if (left0 == lim) k1 = k0 - 1;
                } else {
                    const int ke = off > 0.0 ? k1 : k0;
                    const long long X = XL + static_cast<long long>(ke) * S;
                    if (X > L - T && X < L + T) {
                        AccWalk wk{left0, 0};
                        acc_advance(&wk, off, ke);
                        if (wk.x == lim) {
                            if (off > 0.0) --k1;
                            else ++k0;
                        }
                    }
                }
            }
            const long long width = fix32(right0) - fix32(left0);
            auto at = [&](int k) { return XL + static_cast<long long>(k) * S; };
            // starts a hair below 0 (a few lines at most, but of a ray along the edge)
            auto one = [&](int k) { sum += dd_line(I + k * w, at(k), at(k) + width, n); };
            while (k0 <= k1 && at(k0) < 0) one(k0++);
            while (k0 <= k1 && at(k1) < 0) one(k1--);
            xl = at(k0);
            xr = xl + width;
        }
    }
    const bool any = k0 <= k1;
    if (!any) xl = xr = S = 0;  // reads the first pixels of a line where the others are in step
    // The last start whose footprint ends inside the image, with a margin for
    // the FP32 right edge (within 3e-7 of the fixed-point one).
    const long long last = (static_cast<long long>(n - 1) << 32) - 4096 - (xr - xl);
    const long long span = xr - xl;
    const float width = static_cast<float>(span) * 2.3283064365386963e-10f;  // 2^-32
    const bool wide = __any_sync(0xffffffffu, any && !(width >= 0.001f && width <= 2.0f));
    const float ends = sum;
    const long long start = xl;
    float part;  // a group of lines, in units of half the width
    const float beyond = width - 1.0f, inv = any ? 0.5f / width : 0.0f;
    // A line's four pixels are loaded whether its footprint reaches them or not
    // (the copies have three zeros behind each line), and get the weight 0 where
    // it does not: a ray that an infinity or NaN reached this way is summed
    // again below.
    auto step = [&](const float* __restrict__ line) {
        const float* p = line + static_cast<int>(xl >> 32);
        const float p0 = __ldg(p), p1 = __ldg(p + 1), p2 = __ldg(p + 2), p3 = __ldg(p + 3);
        // what is left of the start's interval: exact, so that the three lengths
        // add up to the width to its own digits, however narrow
        const float d = 2.0f - __uint_as_float(0x3F800000u | (static_cast<unsigned>(xl) >> 9));
        part = fmaf(fminf(width, d), p0 + p1, part);
        part = fmaf(__saturatef(width - d), p1 + p2, part);
        part = fmaf(__saturatef(beyond - d), p2 + p3, part);
        xl += S;
    };
    // the same for a line that some of the warp's rays may not have, and where
    // the image may end inside the footprint (the start may sit a hair past
    // n-1, where the exact one is inside)
    auto step_edge = [&](const float* __restrict__ line, int l) {
        const bool on = l >= k0 && l <= k1;
        const int h = static_cast<int>(xl >> 32), i0 = max(min(h, n - 2), 0);
        const float* p = line + i0;
        const float p0 = __ldg(p), p1 = __ldg(p + 1), p2 = __ldg(p + 2), p3 = __ldg(p + 3);
        const float a = h == i0 ? 1.0f + dd_frac(xl) : 2.0f;
        const float e = fminf(a + width, static_cast<float>(n - i0));
        float t = (fminf(e, 2.0f) - a) * (p0 + p1);
        t = fmaf(__saturatef(e - 2.0f), p1 + p2, t);
        t = fmaf(__saturatef(e - 3.0f), p2 + p3, t);
        t = e > a ? __fdividef(t, e - a) : p0 + p1;
        sum += on ? 0.5f * t : 0.0f;
        xl += on ? S : 0;
    };
    // the lines of any ray of the warp, and those that all its rays have
    const int lo = __reduce_min_sync(0xffffffffu, any ? k0 : 0x7fffffff);
    const int hi = __reduce_max_sync(0xffffffffu, any ? k1 : -1);
    const int in = __reduce_max_sync(0xffffffffu, any ? k0 : -1);
    const int out = __reduce_min_sync(0xffffffffu, any ? k1 : 0x7fffffff);
    const float* line = I + (lo <= hi ? lo : 0) * w;
    const long long ahead = (kDdUnroll - 1) * S;
    if (wide) {
        for (int l = k0; l <= k1; ++l, xl += S) sum += dd_line(I + l * w, xl, xl + span, n);
    } else {
        for (int l = lo; l <= hi; l += kDdUnroll, line += kDdUnroll * w) {
            if (l >= in && l + kDdUnroll - 1 <= out && !__any_sync(0xffffffffu, xl > last || xl + ahead > last)) {
                part = 0.0f;
#pragma unroll
                for (int u = 0; u < kDdUnroll; ++u) step(line + u * w);
                sum = fmaf(part, inv, sum);
            } else {  // lines past the last one read the last one
#pragma unroll
                for (int u = 0; u < kDdUnroll; ++u) step_edge(l + u <= hi ? line + u * w : line, l + u);
            }
        }
    }
    if (is < ns) {
        const float length = static_cast<float>(ux ? fabs(dy / sincos[2 * ia + 1]) : fabs(dx / sincos[2 * ia]));
        if (any && !wide && !isfinite(sum)) {
            sum = ends;
            xl = start;
            for (int l = k0; l <= k1; ++l, xl += S) sum += dd_line(I + l * w, xl, xl + span, n);
        }
        proj[blockIdx.y * proj_stride + ray] = sum * length;
    }
}

// The reference's distance-driven grad in FP64 (T = double), one thread per
// pixel: edges, channel range, lengths and sums with its operations.
template <typename T>
__global__ void __launch_bounds__(kDdThreads)
    fp_dd_grad_kernel(const T* __restrict__ proj, T* __restrict__ img, const double* __restrict__ weights,
                      const double* __restrict__ pos, const int* __restrict__ usex, int ns, int na, int nx,
                      int ny, size_t img_stride, size_t proj_stride)
{
    const long long pix = static_cast<long long>(blockIdx.x) * kDdThreads + threadIdx.x;
    if (pix >= static_cast<long long>(nx) * ny) return;
    const int iy = static_cast<int>(pix / nx), ix = static_cast<int>(pix - static_cast<long long>(iy) * nx);
    const T* P = proj + blockIdx.y * proj_stride;
    const size_t total = static_cast<size_t>(na) * ns;
    static_assert(sizeof(T) == 8, "the FP32 grad is fp_dd_grad_f32");
    T sum = 0;
    for (int ia = 0; ia < na; ++ia) {
        const double* pp = pos + static_cast<size_t>(ia) * nx * 2;
        double mid, left, right;
        if (usex[ia]) {
            const double begin = pp[2 * iy], off = pp[2 * iy + 1];
            mid = __dadd_rn(begin, __dmul_rn(off, static_cast<double>(ix)));
            left = ix == 0 ? mid : __dsub_rn(mid, off);
            right = ix == nx - 1 ? mid : __dadd_rn(mid, off);
        } else {
            const double begin = pp[2 * ix], off = pp[2 * ix + 1];
            mid = __dadd_rn(begin, __dmul_rn(off, static_cast<double>(iy)));
            left = iy == 0 ? mid : __dsub_rn(mid, off);
            right = iy == ny - 1 ? mid : __dadd_rn(mid, off);
        }
        if (left > right) {
            const double t = left;
            left = right;
            right = t;
        }
        const double c0 = ceil(__dsub_rn(left, 0.5)), c1 = floor(__dadd_rn(right, 0.5));
        if (!(c0 >= 0.0)) continue;
        // channels past the sinogram's end add 0: the loop stops there (finite
        // for any input)
        const double last = fmin(c1, static_cast<double>(total - 1 - static_cast<size_t>(ia) * ns));
        const int first = static_cast<int>(fmin(c0, last + 1.0));
        T tmp = 0;
        for (int is = first; static_cast<double>(is) <= last; ++is) {
            const double hi = __dadd_rn(static_cast<double>(is), 0.5), lo = __dsub_rn(static_cast<double>(is), 0.5);
            const double len = __dsub_rn(hi < right ? hi : right, lo > left ? lo : left);
            tmp += len * P[static_cast<size_t>(ia) * ns + is] / 2;
        }
        sum += tmp * weights[ia];
    }
    img[blockIdx.y * img_stride + pix] = static_cast<T>(sum);
}

// ---- FP32 grad with fixed-point decisions ---------------------------------------
// Per (pixel, view) the grad's only discontinuous decisions are
// c0 = ceil(left - 0.5) (the view counts iff c0 >= 0; its first channel) and
// c1 = floor(right + 0.5) (its last channel), left/right = begin + off*k -/+ off
// from the reference's FP64 (view, line) table.  A per-call prologue turns that
// table into 32.32 fixed point; the edges are then exact integer arithmetic
// within (1 + (k+1)/2) * 2^-32 of the exact values, and the reference's FP64
// edges are within 1e-12 of those.  Wherever left - 0.5 or right + 0.5 lies
// within kDdFxGuard (2^-16) of an integer the pair reruns the FP64 decision
// code, so every decision is the reference's.  Overlap lengths come from the
// fixed-point offsets to the first channel, in FP32.
struct DdGradFx {
    long long b, o;  // begin and step of one (view, line), 32.32 fixed point; b == kDdFxBad: use FP64
};
constexpr long long kDdFxBad = -0x7fffffffffffffffLL - 1;
constexpr long long kDdHalf = 1LL << 31;
constexpr unsigned kDdFxGuard = 1u << 16;

__global__ void dd_grad_fx_prep(const double* __restrict__ pos, const double* __restrict__ weights,
                                DdGradFx* __restrict__ fx, float* __restrict__ wf, int na, int nx)
{
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < na) wf[i] = static_cast<float>(weights[i]);
    if (i >= static_cast<long long>(na) * nx) return;
    const double b = pos[2 * i], o = pos[2 * i + 1];
    DdGradFx e{kDdFxBad, 0};
    // |begin|, |off| * nx and the edges stay far inside the 64-bit range
    if (fabs(b) < 1073741824.0 && fabs(o) * (nx + 1) < 1073741824.0)
        e = DdGradFx{__double2ll_rn(b * 4294967296.0), __double2ll_rn(o * 4294967296.0)};
    fx[i] = e;
}

// The reference's FP64 decisions for one (pixel, view): false when the view
// adds nothing; else the first channel, the channel count and the edges
// relative to the first channel.
__device__ __forceinline__ bool dd_grad_decide64(const double* __restrict__ pp, int ux, int ix, int iy, int nx,
                                                 int ny, long long room, int& first, int& cnt, float& lr,
                                                 float& rr)
{
    double mid, left, right;
    if (ux) {
        const double begin = pp[2 * iy], off = pp[2 * iy + 1];
        mid = __dadd_rn(begin, __dmul_rn(off, static_cast<double>(ix)));
        left = ix == 0 ? mid : __dsub_rn(mid, off);
        right = ix == nx - 1 ? mid : __dadd_rn(mid, off);
    } else {
        const double begin = pp[2 * ix], off = pp[2 * ix + 1];
        mid = __dadd_rn(begin, __dmul_rn(off, static_cast<double>(iy)));
        left = iy == 0 ? mid : __dsub_rn(mid, off);
        right = iy == ny - 1 ? mid : __dadd_rn(mid, off);
    }
    if (left > right) {
        const double t = left;
        left = right;
        right = t;
    }
    const double c0 = ceil(__dsub_rn(left, 0.5)), c1 = floor(__dadd_rn(right, 0.5));
    if (!(c0 >= 0.0)) return false;
    const double last = fmin(c1, static_cast<double>(room));
    first = static_cast<int>(fmin(c0, last + 1.0));
    cnt = static_cast<int>(last) - first + 1;
    lr = static_cast<float>(__dsub_rn(left, static_cast<double>(first)));
    rr = static_cast<float>(__dsub_rn(right, static_cast<double>(first)));
    return true;
}

__global__ void __launch_bounds__(kDdThreads)
    fp_dd_grad_f32(const float* __restrict__ proj, float* __restrict__ img, const double* __restrict__ pos,
                   const DdGradFx* __restrict__ fx, const float* __restrict__ wf, const int* __restrict__ usex,
                   int ns, int na, int nx, int ny, size_t img_stride, size_t proj_stride)
{
    const long long pix = static_cast<long long>(blockIdx.x) * kDdThreads + threadIdx.x;
    if (pix >= static_cast<long long>(nx) * ny) return;
    const int iy = static_cast<int>(pix / nx), ix = static_cast<int>(pix - static_cast<long long>(iy) * nx);
    const float* P = proj + blockIdx.y * proj_stride;
    const long long total = static_cast<long long>(na) * ns;
    float sum = 0.0f;
    for (int ia = 0; ia < na; ++ia) {
        const int ux = usex[ia];
        const int line = ux ? iy : ix, k = ux ? ix : iy, kmax = ux ? nx - 1 : ny - 1;
        // channels past the sinogram's end add 0: the loop stops there
        const long long room = total - 1 - static_cast<long long>(ia) * ns;
        const DdGradFx e = fx[static_cast<size_t>(ia) * nx + line];
        int first = 0, cnt = 0;
        float lr = 0.0f, rr = 0.0f;
        bool exact = e.b == kDdFxBad;
        if (!exact) {
            const long long mid = e.b + e.o * k;
            long long left = k == 0 ? mid : mid - e.o, right = k == kmax ? mid : mid + e.o;
            if (left > right) {
                const long long t = left;
                left = right;
                right = t;
            }
            const long long L = left - kDdHalf, R = right + kDdHalf;
            const unsigned lf = static_cast<unsigned>(L), rf = static_cast<unsigned>(R);
            if (lf < kDdFxGuard || lf > 0u - kDdFxGuard || rf < kDdFxGuard || rf > 0u - kDdFxGuard) {
                exact = true;  // an edge within 2^-16 of a decision boundary
            } else {
                const long long c0 = (L >> 32) + 1;  // ceil: the fraction is nonzero here
                const long long c1 = R >> 32;         // floor
                if (c0 < 0) continue;
                const long long last = c1 < room ? c1 : room;
                const long long f = c0 < last + 1 ? c0 : last + 1;
                const long long dl = left - (f << 32), dr = right - (f << 32);
                if (dl <= -(1LL << 38) || dl >= (1LL << 38) || dr <= -(1LL << 38) || dr >= (1LL << 38)) {
                    exact = true;  // a footprint wider than the FP32 offsets' range
                } else {
                    first = static_cast<int>(f);
                    cnt = static_cast<int>(last - f + 1);
                    lr = static_cast<float>(static_cast<int>(dl >> 8)) * 5.9604644775390625e-8f;  // 2^-24
                    rr = static_cast<float>(static_cast<int>(dr >> 8)) * 5.9604644775390625e-8f;
                }
            }
        }
        if (exact && !dd_grad_decide64(pos + static_cast<size_t>(ia) * nx * 2, ux, ix, iy, nx, ny, room, first,
                                       cnt, lr, rr))
            continue;
        const float* row = P + static_cast<size_t>(ia) * ns + first;
        float tmp = 0.0f;
        for (int j = 0; j < cnt; ++j) {
            const float fj = static_cast<float>(j);
            const float len = fminf(fj + 0.5f, rr) - fmaxf(fj - 0.5f, lr);
            tmp = fmaf(len, __ldg(row + j) * 0.5f, tmp);
        }
        sum = fmaf(tmp, wf[ia], sum);
    }
    img[blockIdx.y * img_stride + pix] = sum;
}

// ---- FP32 grad by tiles --------------------------------------------------------
// A pixel-view's term is the integral over [x - o, x + o] (x the pixel's
// position, o the view's |offset|) of the sinogram row read as cells of width 1
// around the channels, halved and weighted.  As a function of x it is linear
// between the positions where an end crosses from cell to cell: two knots a
// channel.  So per (tile, view) the window of channels that the tile reaches is
// staged once as those linear pieces, each from the few cells it covers, and a
// pixel-view is one lookup and one FMA, whatever number of channels it covers.
// With y = x + o - 1/2, j = floor(y) and f = y - j, the right end lies in cell
// j + 1; with m = floor(2 o) and g = 2 o - m, the left end lies in cell j - m
// where f < g, else in cell j - m + 1, and the integral is
//   p[j-m+1] + ... + p[j] + g p[left] + f (p[j+1] - p[left]).
// It is continuous in x, so the position needs no exact decision: it is fixed
// point at the middle of a thread's 8 rows, and FP32 along them, relative to the
// channel nearest there (relative to the window's centre, up to 60 channels away,
// cost digits: 5.5e-7 against 1.8e-7 from FP64 for noise on 64^2).
// Two things of the reference are decided: channels past the row's end read on
// into the next view's row (the staging reads on likewise), and a footprint
// that starts at or before -1/2 adds nothing (tiles that reach there test it
// per pixel, in FP64 within 1e-3 of it).  Pixels at the ends of their line have
// one-sided footprints: dd_grad_border sums those and overwrites them.  A (tile,
// view) with an infinity, NaN or a value beyond 1e30 among its pieces is summed
// pixel by pixel.
//
// CTA: 32 x 64 pixels, 8 of one column per thread, a segment of the views in
// blocks of kDgViews; the next block's channels are loaded into registers
// during a block's sums.  Bound by issue (72 % of the slots) and shared loads
// (69 % of their wavefronts): 720 x 729 -> 512^2 1404 us pixel by pixel
// (fp_dd_grad_f32), 147 us here (185 us with the views, border and sum
// kernels).  A running integral over the window, looked up at both ends, took
// as long and lost the digits of small channels beside a large one.
constexpr int kDgTileX = 32, kDgTileY = 64, kDgRows = 8, kDgViews = 16, kDgThreads = 256;
constexpr float kDgMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low bits

// A view's positions: channel of pixel (along, line) = b + along * o + line * l.
struct DdView {
    long long b, o, l;  // 32.32 fixed point
    float of, lf;       // o and l
    float w;            // the view's weight
    int flags;          // kDgUx: lines are rows; kDgBad: not of this form, or out of range
};
constexpr int kDgUx = 1, kDgBad = 2;

// One warp per view, from the reference's (begin, offset) table of its lines.
__global__ void __launch_bounds__(256)
    dd_grad_views(const double* __restrict__ pos, const double* __restrict__ weights, const int* __restrict__ usex,
                  DdView* __restrict__ views, int na, int n)
{
    const int ia = static_cast<int>((blockIdx.x * 256u + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (ia >= na) return;
    const double* pp = pos + static_cast<size_t>(ia) * n * 2;
    const double b = pp[0], o = pp[1], l = n > 1 ? (pp[2 * (n - 1)] - b) / (n - 1) : 0.0;
    bool ok = fabs(b) < 1048576.0 && fabs(o) < 1048576.0 && fabs(l) < 1048576.0 &&
              fabs(o) * n < 1e9 && fabs(l) * n < 1e9;
    for (int i = lane; i < n; i += 32)
        ok = ok && pp[2 * i + 1] == o && fabs(pp[2 * i] - fma(static_cast<double>(i), l, b)) < 1e-8;
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0)
        views[ia] = DdView{ok ? fix32(b) : 0, ok ? fix32(o) : 0, ok ? fix32(l) : 0, static_cast<float>(o),
                           static_cast<float>(l), static_cast<float>(weights[ia]), (usex[ia] ? kDgUx : 0) | (ok ? 0 : kDgBad)};
}

// A pixel-view by itself, for any view: whether it adds anything, its first
// channel, their count and the footprint's ends relative to the first, from
// integers (in FP64 within 2^-16 of where a channel begins or ends, so that the
// cells of no length that the reference reads are read, and for views not of
// DdView's form).
__device__ __forceinline__ bool dd_grad_one(const DdView& v, const double* __restrict__ pp, int ix, int iy, int n,
                                            long long room, int& first, int& cnt, float& lr, float& rr)
{
    const bool ux = v.flags & kDgUx;
    const int along = ux ? ix : iy, line = ux ? iy : ix;
    const long long mid = v.b + along * v.o + line * v.l;
    long long left = along == 0 ? mid : mid - v.o, right = along == n - 1 ? mid : mid + v.o;
    if (left > right) {
        const long long t = left;
        left = right;
        right = t;
    }
    const long long L = left + kDdHalf, R = right + kDdHalf;
    const unsigned lf = static_cast<unsigned>(L), rf = static_cast<unsigned>(R);
    if ((v.flags & kDgBad) || lf < kDdFxGuard || lf > 0u - kDdFxGuard || rf < kDdFxGuard || rf > 0u - kDdFxGuard)
        return dd_grad_decide64(pp, ux, ix, iy, n, n, room, first, cnt, lr, rr);
    const long long c = L >> 32;  // the left end's cell
    first = static_cast<int>(c);
    cnt = static_cast<int>((R >> 32) - c) + 1;
    lr = static_cast<float>(left - (c << 32)) * 2.3283064365386963e-10f;
    rr = static_cast<float>(right - (c << 32)) * 2.3283064365386963e-10f;
    return c >= 0;
}

// The term of a pixel-view, less the view's weight.
__device__ __forceinline__ float dd_grad_term(const float* __restrict__ P, long long row, long long total, int first,
                                              int cnt, float lr, float rr)
{
    float t = 0.0f;
    for (int c = 0; c < cnt; ++c) {
        const float fc = static_cast<float>(c);
        const float len = fminf(fc + 0.5f, rr) - fmaxf(fc - 0.5f, lr);
        if (row + first + c < total) t = fmaf(len, __ldg(P + row + first + c) * 0.5f, t);
    }
    return t;
}

// A view on a tile.
enum DgMode { kDgSkip, kDgInside, kDgEdge, kDgSlow };
struct DgRec {
    // y - 1/2 of the tile's first column half a row below its fourth row,
    // relative to the window's centre, and its steps: 32.32 fixed point
    long long base, sx, sy;
    float syf;    // sy
    float knot;   // g - 1/2
    float limit;  // footprints with y - 1/2 at or below it add nothing
    int mode;
    int m, ux;  // whole channels of a footprint; whether lines are rows
};
static_assert(sizeof(DgRec) == 48, "16-byte loads");

__device__ __forceinline__ DgRec dg_record(const DdView& v, int tx0, int ty0, int* centre, int* need)
{
    const bool ux = v.flags & kDgUx;
    // the reference pixel (the tile's centre); it may lie outside the image
    const long long cx = tx0 + kDgTileX / 2, cy = ty0 + kDgTileY / 2;
    const long long mid = v.b + (ux ? cx : cy) * v.o + (ux ? cy : cx) * v.l;
    const long long kc = (mid + kDdHalf) >> 32;
    DgRec r;
    r.sx = ux ? v.o : v.l;
    r.sy = ux ? v.l : v.o;
    r.syf = ux ? v.lf : v.of;
    const long long o = v.o < 0 ? -v.o : v.o;
    const float reach = fabsf(v.of);
    r.base = mid - (kc << 32) + o - (1ll << 32) - kDgTileX / 2 * r.sx - (kDgTileY / 2 - 3) * r.sy + (r.sy >> 1);
    r.m = dg_spread(2 * o);
    r.knot = static_cast<float>(static_cast<int>((2 * o - (static_cast<long long>(r.m) << 32)) - kDdHalf)) *
             2.3283064365386963e-10f;
    r.ux = ux;
    // positions of the tile lie within e of the centre
    const float e = fabsf(ux ? v.of : v.lf) * (kDgTileX / 2) + fabsf(r.syf) * (kDgTileY / 2) + 0.51f;
    const float start = -0.5f - fmaxf(fminf(static_cast<float>(kc), 1e6f), -1e6f);  // channel -1/2, from the centre
    r.limit = start + (2.0f * reach - 1.0f);
    // A view whose lines run across its channels (angles outside [0, 2 pi) are
    // not folded) has footprints narrow beside the tile, and a weight to match:
    // positions within the tile in FP32 would cost it digits (5e-5 of the peak
    // against 3e-7).
    const bool across = fabsf(v.lf) > 2.0f * reach;
    if ((v.flags & kDgBad) || across || !dg_fits(e, reach) || kc <= -1000000 || kc >= 0x40000000)
        r.mode = kDgSlow;
    else if (e < start - 0.01f)
        r.mode = kDgSkip;
    else
        r.mode = -e - reach > start + 0.01f ? kDgInside : kDgEdge;
    *centre = static_cast<int>(kc);
    *need = r.mode == kDgInside || r.mode == kDgEdge ? dg_need(e, reach) : -1;
    return r;
}

__global__ void __launch_bounds__(kDgThreads, 3)
    dd_grad_tiles(const float* __restrict__ proj, float* __restrict__ out, const double* __restrict__ pos,
                  const DdView* __restrict__ views, int ns, int na, int n, int segs, int seg_len, size_t out_seg,
                  size_t out_img)
{
    constexpr unsigned kSecond = 2 * kDgHalf * sizeof(float2);  // from a piece before the knot to the one after it
    __shared__ __align__(16) float2 s_piece[kDgViews][2][2 * kDgHalf];
    __shared__ __align__(16) float s_row[8][2 * kDgHalf + 4];  // a warp's channels while it forms the pieces
    __shared__ __align__(16) DgRec s_rec[2][kDgViews];  // the block's and the next one's
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx0 = blockIdx.x * kDgTileX, ty0 = blockIdx.y * kDgTileY;
    const int seg = blockIdx.z % segs, b = blockIdx.z / segs;
    const int vb = seg * seg_len, ve = min(na, vb + seg_len);
    const long long total = static_cast<long long>(na) * ns;
    const float* P = proj + b * static_cast<size_t>(total);
    const int ix = tx0 + lane, iy0 = ty0 + warp * kDgRows;

    // staging: a warp takes views warp and warp + 8 of a block, four channels a lane
    constexpr int kPer = kDgViews / 8;
    static_assert(2 * kDgHalf == 4 * 32 && kDgThreads == 256, "four channels a lane, eight warps");
    float4 ch[kPer];
    int need[kPer];
    auto load = [&](int v0, int buf) {
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const int ia = v0 + warp + 8 * h;
            if (ia >= ve) continue;
            const DdView v = views[ia];
            int kc;
            const DgRec rec = dg_record(v, tx0, ty0, &kc, &need[h]);
            if (lane == 0) s_rec[buf][warp + 8 * h] = rec;
            const long long row = static_cast<long long>(ia) * ns, room = min(total - row, 0x7fffffffll);
            const float half_w = 0.5f * v.w;
            auto one = [&](int i) {
                const int rel = 4 * lane + i - kDgHalf, c = kc + rel;
                return abs(rel) <= need[h] && c >= 0 && c < static_cast<int>(room) ? __ldg(P + row + c) * half_w : 0.0f;
            };
            ch[h] = make_float4(one(0), one(1), one(2), one(3));
        }
    };
    auto stage = [&](int v0, int buf) {
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const int j = warp + 8 * h;
            if (v0 + j >= ve) continue;
            float* row = s_row[warp];
            __syncwarp();
            reinterpret_cast<float4*>(row)[lane] = ch[h];
            if (lane == 0) row[2 * kDgHalf] = 0.0f;
            __syncwarp();
            const int m = s_rec[buf][j].m;
            const float g = s_rec[buf][j].knot + 0.5f;
            bool fine = true;
            // the pieces that the tile's positions can fall in
            for (int i = dg_first_piece(need[h], m) + lane; i < kDgHalf + need[h]; i += 32) {
                const float right = row[i + 1], after = row[i - m + 1], before = row[i - m];
                float sum = m > 0 ? row[i] : 0.0f;
                if (m > 1) sum += after;
                for (int k = i - m + 2; k < i; ++k) sum += row[k];
                const float sa = right - before, sb = right - after;
                const float a = fmaf(0.5f, sa, fmaf(g, before, sum)), b = fmaf(0.5f, sb, fmaf(g, after, sum));
                s_piece[j][0][i] = make_float2(a, sa);  // from f = 1/2
                s_piece[j][1][i] = make_float2(b, sb);
                fine = fine && fabsf(a) + fabsf(sa) < 1e30f && fabsf(b) + fabsf(sb) < 1e30f;
            }
            // an infinity's slope would take its value away again
            if (!__all_sync(0xffffffffu, fine) && lane == 0) s_rec[buf][j].mode = kDgSlow;
        }
    };

    const unsigned pieces = static_cast<unsigned>(__cvta_generic_to_shared(&s_piece[0][0][kDgHalf])) -
                            (__float_as_uint(kDgMagic) << 3);
    float acc[kDgRows] = {};
    load(vb, 0);
    int buf = 0;
    for (int v0 = vb; v0 < ve; v0 += kDgViews, buf ^= 1) {
        const int nv = min(kDgViews, ve - v0);
        stage(v0, buf);
        __syncthreads();
        load(v0 + kDgViews, buf ^ 1);
        float blk[kDgRows] = {};  // this block's sums
        for (int j = 0; j < nv; ++j) {
            const DgRec r = s_rec[buf][j];
            if (r.mode == kDgSkip) continue;
            if (r.mode == kDgSlow) {
                const long long row = static_cast<long long>(v0 + j) * ns;
                const DdView v = views[v0 + j];
                for (int k = 0; k < kDgRows; ++k) {
                    const int iy = iy0 + k;
                    int first, cnt;
                    float lr, rr, t = 0.0f;
                    if (ix < n && iy < n &&
                        dd_grad_one(v, pos + static_cast<size_t>(v0 + j) * n * 2, ix, iy, n, total - 1 - row, first, cnt,
                                    lr, rr))
                        t = dd_grad_term(P, row, total, first, cnt, lr, rr);
#pragma unroll
                    for (int q = 0; q < kDgRows; ++q)  // blk stays in registers
                        if (q == k) blk[q] = fmaf(t, v.w, blk[q]);
                }
                continue;
            }
            // the thread's column between its fourth and fifth row: the nearest
            // channel, and the way past it, so that FP32 holds its rows' positions
            const long long X = r.base + lane * r.sx + warp * kDgRows * r.sy;
            const int J = static_cast<int>((X + kDdHalf) >> 32);
            const float xf = static_cast<float>(static_cast<int>(X)) * 2.3283064365386963e-10f;
            const unsigned at = pieces + j * static_cast<unsigned>(sizeof s_piece[0]) + 8 * J, at2 = at + kSecond;
            const float2 sy = make_float2(r.syf, r.syf), x0 = make_float2(xf, xf);
            auto rows = [&](auto keep) {
#pragma unroll
                for (int k = 0; k < kDgRows; k += 2) {
                    const float2 y = __ffma2_rn(make_float2(k - 3.5f, k - 2.5f), sy, x0);
                    const float2 t = __fadd2_rn(y, make_float2(kDgMagic, kDgMagic));
                    const float2 f = __ffma2_rn(__fadd2_rn(t, make_float2(-kDgMagic, -kDgMagic)),
                                                make_float2(-1.0f, -1.0f), y);
                    float2 p, q;
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                                 : "=f"(p.x), "=f"(p.y) : "r"((f.x < r.knot ? at : at2) + (__float_as_uint(t.x) << 3)));
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                                 : "=f"(q.x), "=f"(q.y) : "r"((f.y < r.knot ? at : at2) + (__float_as_uint(t.y) << 3)));
                    keep(y, k, p, q);
                    blk[k] += fmaf(f.x, p.y, p.x);
                    blk[k + 1] += fmaf(f.y, q.y, q.x);
                }
            };
            if (r.mode == kDgInside) {
                rows([](float2, int, float2&, float2&) {});
            } else {  // footprints that start before the first channel are left out
                const float limit = r.limit - static_cast<float>(J);
                rows([&](float2 y, int k, float2& p, float2& q) {
                    auto on = [&](float yk, int iy) {
                        if (fabsf(yk - limit) < 1e-3f && ix < n && iy < n) {
                            int first, cnt;
                            float lr, rr;
                            return dd_grad_decide64(pos + static_cast<size_t>(v0 + j) * n * 2, r.ux, ix, iy,
                                                    n, n, total - 1 - static_cast<long long>(v0 + j) * ns, first, cnt,
                                                    lr, rr);
                        }
                        return yk > limit;
                    };
                    if (!on(y.x, iy0 + k)) p = make_float2(0.0f, 0.0f);
                    if (!on(y.y, iy0 + k + 1)) q = make_float2(0.0f, 0.0f);
                });
            }
        }
#pragma unroll
        for (int k = 0; k < kDgRows; ++k) acc[k] += blk[k];
        __syncthreads();
    }
    float* O = out + seg * out_seg + b * out_img;
#pragma unroll
    for (int k = 0; k < kDgRows; ++k)
        if (ix < n && iy0 + k < n) O[static_cast<size_t>(iy0 + k) * n + ix] = acc[k];
}

// The 4n - 4 pixels at the image's border, overwriting dd_grad_tiles' values: a
// warp takes 32 adjacent pixels of one side and every 32nd view, so that its
// loads are adjacent channels of a row, and the block's warps are added in a
// fixed order.  Their footprints are one-sided where the pixel ends its line.
constexpr int kDbThreads = 1024;
__global__ void __launch_bounds__(kDbThreads)
    dd_grad_border(const float* __restrict__ proj, float* __restrict__ img, const double* __restrict__ pos,
                   const DdView* __restrict__ views, int ns, int na, int n, int groups)
{
    __shared__ float s_sum[kDbThreads / 32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int side = blockIdx.x / groups, i = (blockIdx.x - side * groups) * 32 + lane;
    const int end = side & 1 ? n - 1 : 0;
    const int ix = side < 2 ? min(i, n - 1) : end, iy = side < 2 ? end : min(i, n - 1);
    const long long total = static_cast<long long>(na) * ns;
    const float* P = proj + blockIdx.y * static_cast<size_t>(total);
    float sum = 0.0f;
    for (int ia = warp; ia < na; ia += kDbThreads / 32) {
        const DdView v = views[ia];
        const long long row = static_cast<long long>(ia) * ns;
        int first, cnt;
        float lr, rr;
        if (!dd_grad_one(v, pos + static_cast<size_t>(ia) * n * 2, ix, iy, n, total - 1 - row, first, cnt, lr, rr)) continue;
        sum = fmaf(dd_grad_term(P, row, total, first, cnt, lr, rr), v.w, sum);
    }
    s_sum[warp][lane] = sum;
    __syncthreads();
    if (warp == 0 && i < n) {
        float a = s_sum[0][lane];
#pragma unroll
        for (int k = 1; k < kDbThreads / 32; ++k) a += s_sum[k][lane];
        img[static_cast<size_t>(blockIdx.y) * n * n + static_cast<size_t>(iy) * n + ix] = a;
    }
}

// img[e] = part[0][e] + part[1][e] + ... in segment order.
__global__ void __launch_bounds__(256)
    dd_grad_sum(const float* __restrict__ part, float* __restrict__ img, size_t count, int segs)
{
    for (size_t e = blockIdx.x * 256ull + threadIdx.x; e < count; e += gridDim.x * 256ull) {
        float a = part[e];
        for (int s = 1; s < segs; ++s) a += part[s * count + e];
        img[e] = a;
    }
}

int check_dd(const ctr_par_param* p, const void* a, const void* b, const void* t0, const void* t1,
             const void* t2, int batch)
{
    if (!p || bad_ptr(a) || bad_ptr(b) || bad_ptr(t0) || bad_ptr(t1) || bad_ptr(t2))
        return fail(CTR_ERR_INVALID_ARG, "null argument");
    int st = check_common(batch);
    if (st) return st;
    if (p->ns < 1 || p->na < 1 || p->nx < 1 || p->ny < 1) return fail(CTR_ERR_INVALID_ARG, "empty geometry");
    if (p->nx != p->ny) return fail(CTR_ERR_INVALID_ARG, "distance-driven projection needs nx == ny");
    if (batch > 65535) return fail(CTR_ERR_UNSUPPORTED, "batch > 65535");
    if (a == b) return fail(CTR_ERR_INVALID_ARG, "projection cannot run in place");
    return CTR_OK;
}

template <typename T>
int dd_forward(const ctr_par_param* p, const T* img, T* proj, const double* sc, const double* bo, const int* usex,
               int batch, cudaStream_t stream)
{
    int st = check_dd(p, img, proj, sc, bo, usex, batch);
    if (st) return st;
    const unsigned long long rays = static_cast<unsigned long long>(p->na) * p->ns;
    const size_t is = static_cast<size_t>(p->nx) * p->ny, ps = static_cast<size_t>(p->na) * p->ns;
    const dim3 grid(div_up(rays, kDdThreads), batch);
    auto by_rays = [&] {
        fp_dd_rays<T><<<grid, kDdThreads, 0, stream>>>(img, proj, sc, bo, usex, p->ns, p->na, p->nx, p->ny, p->dx, p->dy,
                                                       is, ps);
        return check_launch("fp_par_2d distance driven");
    };
    if constexpr (sizeof(T) == 8) {
        return by_rays();
    } else {
        const int n = static_cast<int>(p->nx);
        float* rows = nullptr;
        const size_t copy = static_cast<size_t>(n) * (n + kDdPad);
        int most = batch;  // images at a time: fewer where there is no room for every one's copies
        cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&rows), 2 * sizeof(float) * copy * most, stream);
        while (e == cudaErrorMemoryAllocation && most > 1) {
            cudaGetLastError();
            most = (most + 1) / 2;
            e = cudaMallocAsync(reinterpret_cast<void**>(&rows), 2 * sizeof(float) * copy * most, stream);
        }
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return by_rays();
        }
        if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "distance-driven scratch: %s", cudaGetErrorString(e));
        const unsigned tiles = div_up(n + kDdPad, 32), chunks = div_up(p->ns, kDdRayThreads);
        for (int i = 0; i < batch; i += most) {
            const int count = std::min(most, batch - i);
            float* cols = rows + copy * count;
            dd_copies<<<dim3(tiles, tiles, count), 256, 0, stream>>>(img + i * is, rows, cols, n);
            fp_dd_f32<<<dim3(chunks * p->na, count), kDdRayThreads, 0, stream>>>(
                img + i * is, rows, cols, proj + i * ps, sc, bo, usex, p->ns, chunks, n, p->dx, p->dy, is, ps);
        }
        st = check_launch("fp_par_2d distance driven");
        cudaFreeAsync(rows, stream);  // after the kernel that reads it
        return st;
    }
}

constexpr int kDgNotTiles = -1;

// The grad by tiles, kDgNotTiles where a tile's channels do not fit its window
// (pixels of more than ~1.6 channels): those calls run pixel by pixel.  By
// tiles is the faster one wherever it can run: 512^2 x 720 x 729 185 us against
// 1415, 64^2 x 90 x 96 40 against 76.
int dd_grad_by_tiles(const ctr_par_param* p, const float* proj, float* img, const double* w, const double* pos,
                     const int* usex, int batch, cudaStream_t stream)
{
    const int n = static_cast<int>(p->nx), na = static_cast<int>(p->na);
    const double reach = std::hypot(kDgTileX / 2 * p->dx, kDgTileY / 2 * p->dy) + std::fmax(std::fabs(p->dx), std::fabs(p->dy));
    if (!(reach / std::fabs(p->ds) < kDgHalf - 4)) return kDgNotTiles;
    const int tiles_x = div_up(n, kDgTileX), tiles_y = div_up(n, kDgTileY);
    const long long tiles = static_cast<long long>(tiles_x) * tiles_y;
    // Segments of the views per tile, for the fewest view blocks on the busiest
    // SM (three CTAs a SM).  A function of the geometry and device only, so an
    // image's sums are the same in any batch.
    const int blocks = div_up(na, kDgViews), slots = 3 * device_sms();
    int segs = 1, len = blocks;
    long long best = (tiles + slots - 1) / slots * blocks;
    for (int s = 2; s <= 16 && s <= blocks; ++s) {
        const int l = div_up(blocks, s), used = div_up(blocks, l);
        const long long cost = (tiles * used + slots - 1) / slots * l;
        if (cost < best) {
            best = cost;
            segs = used;
            len = l;
        }
    }
    if (tiles_y > 65535) return kDgNotTiles;
    // Images at a time: as many as the grid takes, fewer where there is no room for
    // their partial images (an image's sums stay the same), and without partial
    // images where there is none for one's.
    const size_t image = static_cast<size_t>(n) * n, part_at = (sizeof(DdView) * na + 255) / 256 * 256;
    int most = std::min(batch, 65535 / segs);
    char* scratch = nullptr;
    while (cudaMallocAsync(reinterpret_cast<void**>(&scratch),
                           part_at + (segs > 1 ? sizeof(float) * segs * image * most : 0), stream) != cudaSuccess) {
        cudaGetLastError();
        if (segs == 1) return kDgNotTiles;
        if (most > 1) {
            most = (most + 1) / 2;
        } else {
            segs = 1;
            len = blocks;
            most = batch;
        }
    }
    DdView* views = reinterpret_cast<DdView*>(scratch);
    dd_grad_views<<<div_up(na, 8), 256, 0, stream>>>(pos, w, usex, views, na, n);
    const int groups = div_up(n, 32);
    for (int i = 0; i < batch; i += most) {
        const int some = std::min(most, batch - i);
        const size_t count = image * some;
        const float* P = proj + static_cast<size_t>(i) * p->na * p->ns;
        float* out = img + i * image;
        float* part = segs > 1 ? reinterpret_cast<float*>(scratch + part_at) : out;
        dd_grad_tiles<<<dim3(tiles_x, tiles_y, segs * some), kDgThreads, 0, stream>>>(
            P, part, pos, views, static_cast<int>(p->ns), na, n, segs, len * kDgViews, count, image);
        if (segs > 1)
            dd_grad_sum<<<std::min<size_t>(div_up(count, 256), 8u * device_sms()), 256, 0, stream>>>(part, out, count, segs);
        dd_grad_border<<<dim3(4 * groups, some), kDbThreads, 0, stream>>>(P, out, pos, views, static_cast<int>(p->ns), na, n,
                                                                         groups);
    }
    const int st = check_launch("fp_par_2d distance-driven grad");
    cudaFreeAsync(scratch, stream);  // after the kernels that read it
    return st;
}

template <typename T>
int dd_grad(const ctr_par_param* p, const T* proj, T* img, const double* w, const double* pos, const int* usex,
            int batch, cudaStream_t stream)
{
    int st = check_dd(p, proj, img, w, pos, usex, batch);
    if (st) return st;
    const unsigned long long pix = static_cast<unsigned long long>(p->nx) * p->ny;
    if constexpr (sizeof(T) == 8) {
        fp_dd_grad_kernel<T><<<dim3(div_up(pix, kDdThreads), batch), kDdThreads, 0, stream>>>(
            proj, img, w, pos, usex, p->ns, p->na, p->nx, p->ny, static_cast<size_t>(p->nx) * p->ny,
            static_cast<size_t>(p->na) * p->ns);
        return check_launch("fp_par_2d distance-driven grad");
    } else {
        const int rc = dd_grad_by_tiles(p, proj, img, w, pos, usex, batch, stream);
        if (rc != kDgNotTiles) return rc;
        // the fixed-point table and FP32 weights of this call (stream-ordered scratch)
        const size_t n_fx = static_cast<size_t>(p->na) * p->nx;
        char* scratch = nullptr;
        cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&scratch),
                                        sizeof(DdGradFx) * n_fx + sizeof(float) * p->na, stream);
        if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "distance-driven grad scratch: %s", cudaGetErrorString(e));
        DdGradFx* fx = reinterpret_cast<DdGradFx*>(scratch);
        float* wf = reinterpret_cast<float*>(fx + n_fx);
        dd_grad_fx_prep<<<div_up(n_fx > p->na ? n_fx : p->na, 256), 256, 0, stream>>>(pos, w, fx, wf, p->na, p->nx);
        fp_dd_grad_f32<<<dim3(div_up(pix, kDdThreads), batch), kDdThreads, 0, stream>>>(
            proj, img, pos, fx, wf, usex, p->ns, p->na, p->nx, p->ny, static_cast<size_t>(p->nx) * p->ny,
            static_cast<size_t>(p->na) * p->ns);
        st = check_launch("fp_par_2d distance-driven grad");
        cudaFreeAsync(scratch, stream);  // after the kernels that read it
        return st;
    }
}

bool dd_views_along_x(double angle)
{
    return !((angle >= kDdPi / 4 && angle < 3 * kDdPi / 4) || (angle >= 5 * kDdPi / 4 && angle < 7 * kDdPi / 4));
}

template <typename V>
int dd_upload(V* dst, const std::vector<V>& src, cudaStream_t stream)
{
    cudaError_t e = cudaMemcpyAsync(dst, src.data(), src.size() * sizeof(V), cudaMemcpyHostToDevice, stream);
    // the host vector dies on return: wait for the staged copy to leave it
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e == cudaSuccess ? CTR_OK : fail(CTR_ERR_CUDA, "distance-driven tables: %s", cudaGetErrorString(e));
}

}  // namespace
}  // namespace ctr

using namespace ctr;

extern "C" {

int ctr_fp_par_2d_dd_prep(const ctr_par_param* p, double* sincostbl, double* beginoffset, int* usex,
                          cudaStream_t stream)
{
    // reference src/fp_par_2d.cc:396-452 (running angle wrapped into [0, 2pi))
    if (!p || bad_ptr(sincostbl) || bad_ptr(beginoffset) || bad_ptr(usex))
        return fail(CTR_ERR_INVALID_ARG, "null argument");
    if (p->na < 1 || p->ns < 1 || p->nx < 1 || p->ny < 1) return fail(CTR_ERR_INVALID_ARG, "empty geometry");
    const double centx = static_cast<double>(p->nx - 1) / 2.0 + p->offset_x;
    const double centy = static_cast<double>(p->ny - 1) / 2.0 + p->offset_y;
    const double cents = static_cast<double>(p->ns - 1) / 2.0 + p->offset_s;
    std::vector<double> sc(2 * static_cast<size_t>(p->na)), bo(static_cast<size_t>(p->na) * p->ns * 3);
    std::vector<int> ux(p->na);
    double angle = p->orbit_start;
    for (unsigned ia = 0; ia < p->na; ++ia) {
        while (angle < 0) angle += 2 * kDdPi;
        while (angle >= 2 * kDdPi) angle -= 2 * kDdPi;
        const double sa = std::sin(angle), ca = std::cos(angle);
        sc[2 * ia] = sa;
        sc[2 * ia + 1] = ca;
        ux[ia] = dd_views_along_x(angle) ? 1 : 0;
        double step, chan, begin;
        if (ux[ia]) {
            step = p->dy * sa / (ca * p->dx);
            chan = p->ds / (ca * p->dx);
            begin = centx - centy * step - cents * chan;
        } else {
            step = p->dx * ca / (sa * p->dy);
            chan = -p->ds / (sa * p->dy);
            begin = centy - centx * step - cents * chan;
        }
        for (unsigned is = 0; is < p->ns; ++is) {
            const size_t r = (static_cast<size_t>(ia) * p->ns + is) * 3;
            bo[r] = begin;
            bo[r + 1] = step;
            bo[r + 2] = chan / 2;
            begin += chan;
        }
        angle += p->orbit;
    }
    int st = dd_upload(sincostbl, sc, stream);
    if (st == CTR_OK) st = dd_upload(beginoffset, bo, stream);
    if (st == CTR_OK) st = dd_upload(usex, ux, stream);
    return st;
}

int ctr_fp_par_2d_dd_grad_prep(const ctr_par_param* p, double* weights, double* pos, int* usex,
                               cudaStream_t stream)
{
    // reference src/fp_par_2d.cc:547-596 (the angle is not wrapped here)
    if (!p || bad_ptr(weights) || bad_ptr(pos) || bad_ptr(usex)) return fail(CTR_ERR_INVALID_ARG, "null argument");
    if (p->na < 1 || p->ns < 1 || p->nx < 1 || p->ny < 1) return fail(CTR_ERR_INVALID_ARG, "empty geometry");
    if (p->nx != p->ny) return fail(CTR_ERR_INVALID_ARG, "distance-driven projection needs nx == ny");
    const double centx = static_cast<double>(p->nx - 1) / 2.0 + p->offset_x;
    const double centy = static_cast<double>(p->ny - 1) / 2.0 + p->offset_y;
    const double cents = static_cast<double>(p->ns - 1) / 2.0 + p->offset_s;
    std::vector<double> w(p->na), ps(static_cast<size_t>(p->na) * p->nx * 2);
    std::vector<int> ux(p->na);
    double angle = p->orbit_start;
    for (unsigned ia = 0; ia < p->na; ++ia) {
        const double sa = std::sin(angle), ca = std::cos(angle);
        ux[ia] = dd_views_along_x(angle) ? 1 : 0;
        double begin, o1, o2;
        if (ux[ia]) {
            w[ia] = std::fabs(p->dy / ca);
            o1 = p->dx * ca / p->ds;
            o2 = -p->dy * sa / p->ds;
            begin = cents - centx * o1 - centy * o2;
        } else {
            w[ia] = std::fabs(p->dx / sa);
            o1 = -p->dy * sa / p->ds;
            o2 = p->dx * ca / p->ds;
            begin = cents - centy * o1 - centx * o2;
        }
        for (unsigned i = 0; i < p->nx; ++i) {
            const size_t r = (static_cast<size_t>(ia) * p->nx + i) * 2;
            ps[r] = begin;
            ps[r + 1] = o1;
            begin += o2;
        }
        angle += p->orbit;
    }
    int st = dd_upload(weights, w, stream);
    if (st == CTR_OK) st = dd_upload(pos, ps, stream);
    if (st == CTR_OK) st = dd_upload(usex, ux, stream);
    return st;
}

int ctr_fp_par_2d_dd_f32(const ctr_par_param* p, const float* img, float* proj, const double* sincostbl,
                         const double* beginoffset, const int* usex, int batch, cudaStream_t stream)
{
    return dd_forward<float>(p, img, proj, sincostbl, beginoffset, usex, batch, stream);
}
int ctr_fp_par_2d_dd_f64(const ctr_par_param* p, const double* img, double* proj, const double* sincostbl,
                         const double* beginoffset, const int* usex, int batch, cudaStream_t stream)
{
    return dd_forward<double>(p, img, proj, sincostbl, beginoffset, usex, batch, stream);
}
int ctr_fp_par_2d_dd_grad_f32(const ctr_par_param* p, const float* proj, float* img, const double* weights,
                              const double* pos, const int* usex, int batch, cudaStream_t stream)
{
    return dd_grad<float>(p, proj, img, weights, pos, usex, batch, stream);
}
int ctr_fp_par_2d_dd_grad_f64(const ctr_par_param* p, const double* proj, double* img, const double* weights,
                              const double* pos, const int* usex, int batch, cudaStream_t stream)
{
    return dd_grad<double>(p, proj, img, weights, pos, usex, batch, stream);
}

}  // extern "C"
