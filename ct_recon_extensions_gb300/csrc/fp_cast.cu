// Ray-casting parallel forward projection: the reference's
// ParallelProjection2DRayCasting (src/fp_par_2d.cc:18-145).
//
// A ray enters the FoV circle (radius fov) at (x1, y1) in pixel-index units
// and takes nsteps samples of step step_size pixels along (sin t, cos t); a
// sample at the FP64 running position (x1 + sx + sx + ..., y1 + sy + ...) is
// used iff 0 <= x <= nx-1 and 0 <= y <= ny-1, and adds the bilinear
// interpolation of its four neighbours (floor / ceil corners).  The ray sum is
// scaled by step_size * dx.
//
// FP32 path (fp_cast_rows_f32 for steps up to half a pixel, fp_cast_f32 above and
// where an image's copies do not fit).  The sample range of each axis is decided
// exactly as the reference decides it: in 32.32 fixed point where that is certain,
// and by the reference's own FP64 accumulation (acc_advance, jumping binade to
// binade) for the few samples within a hair of an image edge (fp_setup.cuh).  The
// running position is monotone in k, so each axis keeps a contiguous range and the
// ray keeps their intersection.  Inside it both coordinates are fixed point and the
// interpolation FP32; positions differ from the reference's FP64 ones by ~1e-9
// pixel, which moves the interpolation weights by as much (continuous at pixel
// boundaries).
//
// FP64 path: one thread per ray, the reference's loop (FP64 positions and
// inclusion test, FP64 interpolation and sum).
#include <algorithm>
#include <cmath>
#include <vector>

#include "ctr_common.cuh"
#include "fp_setup.cuh"

namespace ctr {
namespace {

constexpr int kCastThreads = 128;

// Fraction of a 32.32 fixed-point value, from its low word's top 23 bits.
__device__ __forceinline__ float cast_frac(long long X)
{
    return __uint_as_float(0x3F800000u | (static_cast<unsigned>(X) >> 9)) - 1.0f;
}

// The FP32 kernel: a warp takes 32 consecutive rays.  Each lane first sets up
// one of them (sample range and fixed-point lines), then the warp marches the
// rays one after the other, lane l taking samples k0 + l, k0 + l + 32, ...: a
// warp's 32 samples lie within ~4 pixels of each other, so the four corner
// loads of a step touch a couple of cache lines instead of 32.  Each lane sums
// its samples in FP32, and a fixed shuffle tree adds the 32 lane sums.
__global__ void __launch_bounds__(kCastThreads)
    fp_cast_f32(const float* __restrict__ img, float* __restrict__ proj, const double* __restrict__ sincos,
                const double* __restrict__ begins, const int* __restrict__ nsteps, int ns, int na, int nx,
                int ny, double step_size, float scale, size_t img_stride, size_t proj_stride)
{
    const long long rays = static_cast<long long>(na) * ns;
    const int lane = threadIdx.x & 31;
    const long long r0 = (static_cast<long long>(blockIdx.x) * kCastThreads + threadIdx.x) - lane;
    if (r0 >= rays) return;  // warp-uniform
    // ---- set-up: lane l, ray r0 + l
    const long long ray = r0 + lane;
    long long X0 = 0, SX = 0, Y0 = 0, SY = 0;
    int k0 = 0, k1 = -1;
    if (ray < rays) {
        const int nstep = nsteps[ray];
        if (nstep > 0) {
            const int ia = static_cast<int>(ray / ns);
            const double sx = step_size * sincos[2 * ia], sy = step_size * sincos[2 * ia + 1];
            int kx0, kx1, ky0, ky1;
            axis_range(begins[2 * ray], sx, nstep, nx, &X0, &SX, &kx0, &kx1);
            axis_range(begins[2 * ray + 1], sy, nstep, ny, &Y0, &SY, &ky0, &ky1);
            k0 = max(kx0, ky0);
            k1 = min(kx1, ky1);
        }
    }
    const float* I = img + blockIdx.y * img_stride;
    float* out = proj + blockIdx.y * proj_stride;
    const int nr = static_cast<int>(min(32ll, rays - r0));
    for (int j = 0; j < nr; ++j) {
        const int a = __shfl_sync(0xffffffffu, k0, j), b = __shfl_sync(0xffffffffu, k1, j);
        const long long xs = __shfl_sync(0xffffffffu, SX, j), ys = __shfl_sync(0xffffffffu, SY, j);
        long long x = __shfl_sync(0xffffffffu, X0, j) + static_cast<long long>(a + lane) * xs;
        long long y = __shfl_sync(0xffffffffu, Y0, j) + static_cast<long long>(a + lane) * ys;
        const long long xs32 = xs * 32, ys32 = ys * 32;
        float part = 0.0f;
        for (int k = a + lane; k <= b; k += 32) {
            // exact positions are inside; the fixed-point ones may sit a hair
            // outside an edge: clamp the corner (the weight there is ~0)
            const int xi = static_cast<int>(x >> 32), yi = static_cast<int>(y >> 32);
            const int ix = min(max(xi, 0), nx - 1), iy = min(max(yi, 0), ny - 1);
            const float u = xi == ix ? cast_frac(x) : 0.0f, v = yi == iy ? cast_frac(y) : 0.0f;
            const int ix2 = min(ix + 1, nx - 1);
            const float* q1 = I + static_cast<size_t>(iy) * nx;
            const float* q2 = I + static_cast<size_t>(min(iy + 1, ny - 1)) * nx;
            const float a0 = __ldg(q1 + ix), a1 = __ldg(q1 + ix2);
            const float b0 = __ldg(q2 + ix), b1 = __ldg(q2 + ix2);
            const float p = fmaf(u, a1 - a0, a0), q = fmaf(u, b1 - b0, b0);
            part += fmaf(v, q - p, p);
            x += xs32;
            y += ys32;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == j) out[r0 + j] = part * scale;
    }
}

// ---- FP32, small steps: one closed form per image row ------------------------
// A ray marched along its steeper axis takes 1 / (|sin| or |cos| * step_size)
// samples between two image rows, and crosses at most one column boundary on
// the way.  The bilinear interpolant is (1 - v) P_j(x) + v P_j+1(x) there, each
// P piecewise linear with its one knot at that boundary, and the samples are
// arithmetic progressions in x and v, so their sum is six pixels with weights
// that the sums of 1, k and k^2 over the samples before and after the knot
// give: the work is per row crossed (9.3 samples a row on average at a step of
// 0.125 pixel) instead of per sample.  A sample put on the wrong side of a row
// or of the knot lies within FP32 rounding of it, where both forms agree.
//
// One lane per ray, a block's lanes on adjacent channels of one view, so a
// warp's pixels of a row are adjacent; rays marched in x read the transposed
// copy.  Both copies have a border of kCastPad zeros around the image (the
// fixed-point positions may sit a hair outside it, where the weight is ~0), so
// the loop has no clamps.  Issue bound: ~75 instructions per ray and row, 66 %
// of the issue slots (512^2 x 720 x 729 at a step of 0.125: 2450 -> 403 us).
// Blocks start with the long rays of every view, near the detector's middle, and
// end with short ones: view by view the SMs ran dry one by one (467 us).
// Blocks of 64 rays took 411 us, of 128 422; fewer registers for more warps
// spilled (20 blocks of 64 a SM, view by view: 526 us).
//
// A row's six products are one number, rows are added kCastFold at a time, and
// what the total cannot hold of these goes to the next ones: 3.7e-8 from FP64 for
// phantoms on 128^2 to 300^2, 1.0e-7 for noise (sample by sample 4e-8 to 2e-7 by
// the step; six running sums over all rows 2.3e-7, and 394 us).  Lanes are brought
// together only there.
constexpr int kCastPad = 2;
constexpr int kRowThreads = 32, kRowBlocks = 32;  // rays a block, blocks an SM
constexpr int kCastFold = 8;                      // rows summed by themselves

// The padded image and its padded transpose, 32 x 32 tiles of padded pixels.
__global__ void __launch_bounds__(256)
    cast_pad(const float* __restrict__ img, float* __restrict__ rows, float* __restrict__ cols, int nx, int ny)
{
    __shared__ float t[32][33];
    const int wx = nx + 2 * kCastPad, wy = ny + 2 * kCastPad;
    const size_t off = static_cast<size_t>(blockIdx.z) * nx * ny, poff = static_cast<size_t>(blockIdx.z) * wx * wy;
    const int x0 = blockIdx.x * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    // grid.y strides over the rows of tiles
    for (int y0 = blockIdx.y * 32; y0 < wy; y0 += gridDim.y * 32) {
        for (int r = ty; r < 32; r += 8) {
            const int x = x0 + tx - kCastPad, y = y0 + r - kCastPad;
            const float v = x >= 0 && x < nx && y >= 0 && y < ny ? img[off + static_cast<size_t>(y) * nx + x] : 0.0f;
            t[r][tx] = v;
            if (x0 + tx < wx && y0 + r < wy) rows[poff + static_cast<size_t>(y0 + r) * wx + x0 + tx] = v;
        }
        __syncthreads();
        for (int r = ty; r < 32; r += 8)
            if (x0 + r < wx && y0 + tx < wy) cols[poff + static_cast<size_t>(x0 + r) * wy + y0 + tx] = t[tx][r];
        __syncthreads();
    }
}

// The bits of 1 + the fraction of a 32.32 fixed-point value (its top 23 bits).
__device__ __forceinline__ float cast_one_frac(unsigned long long X)
{
    return __uint_as_float(0x3F800000u | (static_cast<unsigned>(X) >> 9));
}

// One lane's ray of the row-by-row march: its first sample and step on the
// marched axis (M, MS) and across it (C, CS; mirrored where the ray runs down
// the image, so that CS >= 0), both 32.32 fixed point, and its samples.
struct CastRay {
    unsigned long long M, C;
    unsigned MS, CS;  // below 1 pixel
    int left;
};

// The sum over a ray's samples; the warp's lanes take the image rows together
// (a lane waits for the row its ray starts on), so that each load reads
// adjacent pixels of one row.  P: the copy, at pixel (0, 0); w: its row stride;
// Dir: the direction of C in the image.
template <int Dir>
__device__ __forceinline__ float cast_march(CastRay r, const float* __restrict__ P, int w)
{
    const float a = static_cast<float>(r.CS) * 2.3283064365386963e-10f;  // 2^-32
    const float b = static_cast<float>(r.MS) * 2.3283064365386963e-10f;
    const float inv_a = __fdividef(1.0f, a), inv_b = __fdividef(1.0f, b);
    const float nab3 = a * b * (-1.0f / 3.0f);
    const float2 a2 = make_float2(a, a), nab2 = make_float2(nab3, nab3);
    const float2 half2 = make_float2(0.5f, 0.5f), mhalf2 = make_float2(-0.5f, -0.5f);
    const float2 two2 = make_float2(2.0f, 2.0f), minus1 = make_float2(-1.0f, -1.0f);
    float sum = 0.0f, part = 0.0f;  // all rows, and the last ones
    int j = __reduce_min_sync(0xffffffffu, r.left > 0 ? static_cast<int>(r.M >> 32) : 0x7fffffff);
    while (__any_sync(0xffffffffu, r.left > 0)) {
        for (const int end = j + kCastFold; j < end; ++j) {
            const int row = static_cast<int>(r.M >> 32), col = static_cast<int>(r.C >> 32);
            if (r.left <= 0 || row > j) continue;
            const float* p = P + (Dir > 0 ? row * w + col : row * w - col);
            const float* p1 = p + w;
            const float v1 = cast_one_frac(r.M), u1 = cast_one_frac(r.C);
            const float d0 = 2.0f - u1, v0 = v1 - 1.0f;  // distance to the knot, position past the row
            // samples in this row, and those of them before the knot
            const int m = min(r.left, __float2int_ru((2.0f - v1) * inv_b));  // >= 1: v1 < 2
            const int q = min(m, __float2int_ru(d0 * inv_a));
            const float2 B = make_float2(__ldg(p), __ldg(p1));
            const float2 K = make_float2(__ldg(p + Dir), __ldg(p1 + Dir));
            float2 A = make_float2(0.0f, 0.0f);  // past the knot: only where a sample is
            if (q < m) A = make_float2(__ldg(p + 2 * Dir), __ldg(p1 + 2 * Dir));
            // over the first q and over all m samples, packed: x, the sum of the
            // positions past the knot -d0 + k a, and y, minus the sum of v times it
            // (v = v0 + k b)
            const float2 n = make_float2(static_cast<float>(q), static_cast<float>(m));
            const float2 s1 = __fmul2_rn(n, __ffma2_rn(n, half2, mhalf2));
            const float2 s3 = __fmul2_rn(s1, __ffma2_rn(n, two2, minus1));
            const float vd = v0 * d0, cr = fmaf(d0, b, -v0 * a);
            const float2 x = __ffma2_rn(a2, s1, __fmul2_rn(n, make_float2(-d0, -d0)));
            const float2 y = __ffma2_rn(nab2, s3, __ffma2_rn(make_float2(cr, cr), s1, __fmul2_rn(n, make_float2(vd, vd))));
            const float sv = fmaf(b, s1.y, n.y * v0);  // sum of v
            // weights of the pixel before the knot, after it and at it, rows j and j + 1
            const float2 wb = make_float2(-y.x - x.x, y.x);
            const float wa1 = y.x - y.y;
            const float2 wa = make_float2((x.y - x.x) - wa1, wa1);
            const float2 wk = make_float2((n.y - sv) - wb.x - wa.x, sv - wb.y - wa.y);
            const float2 v = __ffma2_rn(wk, K, __ffma2_rn(wa, A, __fmul2_rn(wb, B)));
            part += v.x + v.y;
            r.left -= m;
            r.M += static_cast<unsigned long long>(static_cast<unsigned>(m)) * r.MS;
            r.C += static_cast<unsigned long long>(static_cast<unsigned>(m)) * r.CS;
        }
        const float t = sum + part;
        part = fabsf(t) <= 3.4e38f ? part - (t - sum) : 0.0f;  // what the sum cannot hold stays
        sum = t;
    }
    return sum + part;
}

__global__ void __launch_bounds__(kRowThreads, kRowBlocks)
    fp_cast_rows_f32(const float* __restrict__ rows, const float* __restrict__ cols, float* __restrict__ proj,
                     const double* __restrict__ sincos, const double* __restrict__ begins,
                     const int* __restrict__ nsteps, int ns, int nx, int ny, unsigned chunks, double step_size,
                     float scale, size_t proj_stride)
{
    // the chunks of channels from the detector's middle outwards, each for every view
    const unsigned na = gridDim.x / chunks, rank = blockIdx.x / na, ia = blockIdx.x - rank * na;
    const unsigned chunk = rank & 1 ? chunks / 2 - (rank + 1) / 2 : chunks / 2 + rank / 2;
    const int is = static_cast<int>(chunk * kRowThreads + threadIdx.x);
    const size_t ray = static_cast<size_t>(ia) * ns + is;
    const double sx = step_size * sincos[2 * ia], sy = step_size * sincos[2 * ia + 1];
    // a view's rays are marched along one axis, turned so that M runs up
    const bool along_y = fabs(sy) >= fabs(sx);
    const bool turn = (along_y ? sy : sx) < 0.0, down = ((along_y ? sx : sy) < 0.0) != turn;
    CastRay r{0, 0, 0, 0, 0};
    if (is < ns) {
        const int nstep = nsteps[ray];
        if (nstep > 0) {
            int kx0, kx1, ky0, ky1;
            long long X, SX, Y, SY;
            axis_range(begins[2 * ray], sx, nstep, nx, &X, &SX, &kx0, &kx1);
            axis_range(begins[2 * ray + 1], sy, nstep, ny, &Y, &SY, &ky0, &ky1);
            const int k0 = max(kx0, ky0), k1 = min(kx1, ky1), ks = turn ? k1 : k0;
            r.left = max(0, k1 - k0 + 1);
            const long long ms = along_y ? SY : SX, cs = along_y ? SX : SY;
            const long long c = (along_y ? X : Y) + ks * cs;
            r.M = (along_y ? Y : X) + ks * ms;
            r.MS = static_cast<unsigned>(turn ? -ms : ms);
            r.C = down ? -c : c;
            r.CS = static_cast<unsigned>(down != turn ? -cs : cs);
        }
    }
    const int w = (along_y ? nx : ny) + 2 * kCastPad;
    const float* P = (along_y ? rows : cols) +
                     static_cast<size_t>(blockIdx.y) * (nx + 2 * kCastPad) * (ny + 2 * kCastPad) +
                     static_cast<size_t>(kCastPad) * w + kCastPad;
    const float sum = down ? cast_march<-1>(r, P, w) : cast_march<1>(r, P, w);
    if (is < ns) proj[blockIdx.y * proj_stride + ray] = sum * scale;
}

__global__ void __launch_bounds__(kCastThreads)
    fp_cast_f64(const double* __restrict__ img, double* __restrict__ proj, const double* __restrict__ sincos,
                const double* __restrict__ begins, const int* __restrict__ nsteps, int ns, int na, int nx,
                int ny, double step_size, double dx, size_t img_stride, size_t proj_stride)
{
    const long long ray = static_cast<long long>(blockIdx.x) * kCastThreads + threadIdx.x;
    if (ray >= static_cast<long long>(na) * ns) return;
    const int ia = static_cast<int>(ray / ns);
    double* out = proj + blockIdx.y * proj_stride + ray;
    const int nstep = nsteps[ray];
    if (nstep <= 0) {
        *out = 0.0;
        return;
    }
    const double sx = step_size * sincos[2 * ia], sy = step_size * sincos[2 * ia + 1];
    const double xmax = static_cast<double>(nx - 1), ymax = static_cast<double>(ny - 1);
    const double* I = img + blockIdx.y * img_stride;
    double x = begins[2 * ray], y = begins[2 * ray + 1], sum = 0.0;
    for (int k = 0; k < nstep; ++k) {
        if (x >= 0 && x <= xmax && y >= 0 && y <= ymax) {
            const int ix1 = static_cast<int>(floor(x)), ix2 = static_cast<int>(ceil(x));
            const int iy1 = static_cast<int>(floor(y)), iy2 = static_cast<int>(ceil(y));
            const double u = x - ix1, v = y - iy1;
            const double* r1 = I + static_cast<size_t>(iy1) * nx;
            const double* r2 = I + static_cast<size_t>(iy2) * nx;
            sum += (1 - v) * ((1 - u) * r1[ix1] + u * r1[ix2]) + v * ((1 - u) * r2[ix1] + u * r2[ix2]);
        }
        x += sx;
        y += sy;
    }
    *out = sum * step_size * dx;
}

int check_cast(const ctr_par_param* p, double step_size, const void* a, const void* b, const void* sc,
               const void* begins, const void* nsteps, int batch)
{
    if (!p || bad_ptr(a) || bad_ptr(b) || bad_ptr(sc) || bad_ptr(begins) || bad_ptr(nsteps))
        return fail(CTR_ERR_INVALID_ARG, "null argument");
    int st = check_common(batch);
    if (st) return st;
    if (p->ns < 1 || p->na < 1 || p->nx < 1 || p->ny < 1) return fail(CTR_ERR_INVALID_ARG, "empty geometry");
    if (!(step_size > 0.0)) return fail(CTR_ERR_INVALID_ARG, "step_size must be positive");
    if (batch > 65535) return fail(CTR_ERR_UNSUPPORTED, "batch > 65535");
    if (a == b) return fail(CTR_ERR_INVALID_ARG, "projection cannot run in place");
    return CTR_OK;
}

// Steps up to this many pixels go row by row (fp_cast_rows_f32): the time does
// not depend on the step there, that of the sample-by-sample kernel does.  Per
// call (copies included), row by row against sample by sample:
//   512^2 x 720 x 729   step 0.125: 403 / 2450 us, 0.5: 403 / 1176
//   128^2 x 180 x 190   step 0.125: 51 / 135 us,   0.5: 41 / 57
//   64^2 x 90 x 96      step 0.125: 34 / 70 us,    0.5: 30 / 33
// (At 0.75 the larger two would gain too, 403 / 1040 and 40 / 45, the last would
// not, 31 / 28: those steps are left sample by sample.)
// Geometries of fewer samples than kCastRowSamples (rays times the image's shorter
// side in steps; an item's path is the same in any batch) are launches, of which the
// copies are one more: 32^2 x 30 x 45 at a step of 0.25 23 / 19 us, 16^2 x 12 x 21
// 21 / 15.  Where the call allocates the copies itself, a synchronisation between
// calls has the pool give the memory back, and the next call takes ~170 us to get
// it: kCastOwnSamples (341^2 x 457 x 424 at 0.125, 5e8: 344 / 900 us with such a
// synchronisation; 183^2 x 255 x 267 at 0.5, 2.5e7: 256 / 95).
constexpr double kCastRowStep = 0.5, kCastRowSamples = 5e5, kCastOwnSamples = 2e8;
constexpr size_t kCastOwnBytes = 256u << 20;  // copies at a time of a call that allocates them

// Bytes of an image's two copies; 0 where an FP32 call goes sample by sample.
size_t cast_copies(const ctr_par_param* p, double step_size, double samples)
{
    const size_t wx = static_cast<size_t>(p->nx) + 2 * kCastPad, wy = static_cast<size_t>(p->ny) + 2 * kCastPad;
    // the march indexes a copy with 32-bit integers
    if (step_size > kCastRowStep || wx * wy > 0x7fffffffu ||
        static_cast<size_t>(div_up(p->ns, kRowThreads)) * p->na > 0x7fffffffu)
        return 0;
    if (static_cast<double>(p->na) * p->ns * std::min(p->nx, p->ny) < samples * step_size) return 0;
    return 2 * sizeof(float) * wx * wy;
}

// An FP32 call row by row, `most` images at a time with their copies in `scratch`.
int cast_rows(const ctr_par_param* p, double step_size, const float* img, float* proj, const double* sc,
              const double* begins, const int* nsteps, int batch, float* scratch, int most, cudaStream_t stream)
{
    const int nx = static_cast<int>(p->nx), ny = static_cast<int>(p->ny);
    const unsigned wx = p->nx + 2 * kCastPad, wy = p->ny + 2 * kCastPad, chunks = div_up(p->ns, kRowThreads);
    const size_t is = static_cast<size_t>(nx) * ny, ps = static_cast<size_t>(p->na) * p->ns;
    for (int i = 0; i < batch; i += most) {
        const unsigned count = std::min(most, batch - i);
        float* cols = scratch + static_cast<size_t>(wx) * wy * count;
        cast_pad<<<dim3(div_up(wx, 32), std::min(div_up(wy, 32), 32768u), count), 256, 0, stream>>>(img + i * is, scratch,
                                                                                                    cols, nx, ny);
        fp_cast_rows_f32<<<dim3(chunks * p->na, count), kRowThreads, 0, stream>>>(
            scratch, cols, proj + i * ps, sc, begins, nsteps, p->ns, nx, ny, chunks, step_size,
            static_cast<float>(step_size * p->dx), ps);
    }
    return check_launch("fp_par_2d ray casting");
}

// The row-by-row path with copies of the call's own; false where there is none, or
// no room for one image's.
bool cast_own_rows(const ctr_par_param* p, double step_size, const float* img, float* proj, const double* sc,
                   const double* begins, const int* nsteps, int batch, cudaStream_t stream, int* status)
{
    const size_t item = cast_copies(p, step_size, kCastOwnSamples);
    if (item == 0) return false;
    int most = static_cast<int>(std::max<size_t>(1, std::min<size_t>(batch, kCastOwnBytes / item)));
    float* scratch = nullptr;
    while (cudaMallocAsync(reinterpret_cast<void**>(&scratch), item * most, stream) != cudaSuccess) {
        cudaGetLastError();
        if (most == 1) return false;
        most = (most + 1) / 2;
    }
    *status = cast_rows(p, step_size, img, proj, sc, begins, nsteps, batch, scratch, most, stream);
    cudaFreeAsync(scratch, stream);  // after the kernel that reads it
    return true;
}

template <typename T>
int cast_forward(const ctr_par_param* p, double step_size, const T* img, T* proj, const double* sc,
                 const double* begins, const int* nsteps, int batch, cudaStream_t stream, bool own = true,
                 void* scratch = nullptr, size_t bytes = 0)
{
    int st = check_cast(p, step_size, img, proj, sc, begins, nsteps, batch);
    if (st) return st;
    const long long rays = static_cast<long long>(p->na) * p->ns;
    const dim3 grid(static_cast<unsigned>(div_up(static_cast<unsigned long long>(rays), kCastThreads)), batch);
    const size_t is = static_cast<size_t>(p->nx) * p->ny, ps = static_cast<size_t>(p->na) * p->ns;
    if constexpr (sizeof(T) == 4) {
        if (own && cast_own_rows(p, step_size, img, proj, sc, begins, nsteps, batch, stream, &st)) return st;
        const size_t item = cast_copies(p, step_size, kCastRowSamples);
        if (item > 0 && bytes >= item)
            return cast_rows(p, step_size, img, proj, sc, begins, nsteps, batch, static_cast<float*>(scratch),
                             static_cast<int>(std::min<size_t>(batch, bytes / item)), stream);
        fp_cast_f32<<<grid, kCastThreads, 0, stream>>>(img, proj, sc, begins, nsteps, p->ns, p->na, p->nx, p->ny, step_size,
                                                       static_cast<float>(step_size * p->dx), is, ps);
    } else
        fp_cast_f64<<<grid, kCastThreads, 0, stream>>>(img, proj, sc, begins, nsteps, p->ns, p->na, p->nx, p->ny,
                                                       step_size, p->dx, is, ps);
    return check_launch("fp_par_2d ray casting");
}

}  // namespace
}  // namespace ctr

using namespace ctr;

extern "C" {

int ctr_fp_par_2d_cast_prep(const ctr_par_param* p, double step_size, double* sincostbl, double* begins,
                            int* nsteps, cudaStream_t stream)
{
    // reference src/fp_par_2d.cc:18-80: running angle and channel coordinate
    // (angle += orbit, s += ds), the angle not wrapped
    if (!p || bad_ptr(sincostbl) || bad_ptr(begins) || bad_ptr(nsteps))
        return fail(CTR_ERR_INVALID_ARG, "null argument");
    if (p->na < 1 || p->ns < 1 || p->nx < 1 || p->ny < 1) return fail(CTR_ERR_INVALID_ARG, "empty geometry");
    if (!(step_size > 0.0)) return fail(CTR_ERR_INVALID_ARG, "step_size must be positive");
    const double xc = static_cast<double>(p->nx - 1) / 2.0 + p->offset_x;
    const double yc = static_cast<double>(p->ny - 1) / 2.0 + p->offset_y;
    const double fov2 = p->fov * p->fov;
    const double s0 = -(static_cast<double>(p->ns - 1) / 2.0 + p->offset_s) * p->ds;
    const size_t rays = static_cast<size_t>(p->na) * p->ns;
    std::vector<double> sc(2 * static_cast<size_t>(p->na)), bg(2 * rays);
    std::vector<int> nst(rays);
    double angle = p->orbit_start;
    for (unsigned ia = 0; ia < p->na; ++ia) {
        const double sa = std::sin(angle), ca = std::cos(angle);
        sc[2 * ia] = sa;
        sc[2 * ia + 1] = ca;
        const double sx = step_size * sa, sy = step_size * ca;
        const bool along_x = sa > (1.0 / 1.414);
        double s = s0;
        for (unsigned is = 0; is < p->ns; ++is) {
            const size_t r = static_cast<size_t>(ia) * p->ns + is;
            const double h2 = fov2 - s * s;
            if (h2 > 0) {
                const double h = std::sqrt(h2);
                const double x1 = (s * ca - h * sa) / p->dx + xc;
                const double y1 = -(s * sa + h * ca) / p->dy + yc;
                const double x2 = (s * ca + h * sa) / p->dx + xc;
                const double y2 = -(s * sa - h * ca) / p->dy + yc;
                nst[r] = along_x ? static_cast<int>((x2 - x1) / sx) : static_cast<int>((y2 - y1) / sy);
                bg[2 * r] = x1;
                bg[2 * r + 1] = y1;
            } else {
                nst[r] = 0;
                bg[2 * r] = 0;
                bg[2 * r + 1] = 0;
            }
            s += p->ds;
        }
        angle += p->orbit;
    }
    cudaError_t e = cudaMemcpyAsync(sincostbl, sc.data(), sc.size() * sizeof(double), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(begins, bg.data(), bg.size() * sizeof(double), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(nsteps, nst.data(), nst.size() * sizeof(int), cudaMemcpyHostToDevice, stream);
    // the host vectors die on return: wait for the staged copies to leave them
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "ray-casting tables: %s", cudaGetErrorString(e));
    return CTR_OK;
}

int ctr_fp_par_2d_cast_f32(const ctr_par_param* p, double step_size, const float* img, float* proj,
                           const double* sincostbl, const double* begins, const int* nsteps, int batch,
                           cudaStream_t stream)
{
    return cast_forward<float>(p, step_size, img, proj, sincostbl, begins, nsteps, batch, stream);
}

size_t ctr_fp_par_2d_cast_scratch(const ctr_par_param* p, double step_size)
{
    return p && p->nx > 0 && p->ny > 0 && step_size > 0.0 ? cast_copies(p, step_size, kCastRowSamples) : 0;
}

int ctr_fp_par_2d_cast_f32_scratch(const ctr_par_param* p, double step_size, const float* img, float* proj,
                                   const double* sincostbl, const double* begins, const int* nsteps, int batch,
                                   void* scratch, size_t bytes, cudaStream_t stream)
{
    if (bytes > 0 && (bad_ptr(scratch) || reinterpret_cast<uintptr_t>(scratch) % sizeof(float) != 0))
        return fail(CTR_ERR_INVALID_ARG, "scratch null or not aligned to a float");
    return cast_forward<float>(p, step_size, img, proj, sincostbl, begins, nsteps, batch, stream, false, scratch, bytes);
}

int ctr_fp_par_2d_cast_f64(const ctr_par_param* p, double step_size, const double* img, double* proj,
                           const double* sincostbl, const double* begins, const int* nsteps, int batch,
                           cudaStream_t stream)
{
    return cast_forward<double>(p, step_size, img, proj, sincostbl, begins, nsteps, batch, stream);
}

}  // extern "C"
