// Fan weighting and ramp filtering (reference src/fan_weighting.cc:19-59,
// src/filter.cc:67-124).
//
// Fan weighting is a diagonal scaling: a CTA computes the FP64 weights of its
// channels once and streams a run of rows; the results are those of the
// reference's FP64 products, bit for bit, for both T.
//
// The ramp filter is a linear (zero-padded) convolution with 2ns+1 taps.  A
// CTA stages kRows rows and the taps in shared memory; each thread produces
// one output column for all staged rows, so a tap load is shared by kRows
// multiply-adds.  The reference kernels have zero even taps (k != 0); when
// the caller's table has that structure (checked in-kernel) only the odd
// taps are visited.
//
// FP32 accuracy: the ramp taps sum to almost zero, so on a smooth sinogram
// the output is a small difference of large partial sums.  The FP32 kernel
// therefore accumulates h[o-j] (x[j] - c) with c a value of the row near the
// thread's outputs, and adds back c (h[0] + sum of the taps that output o
// sums):
//   out[o] = h[0] (x[o] - c) + c D[o] + sum_j h[o-j] (x[j] - c),
//   D[o] = h[0] + sum_{j of the other parity} h[o-j]
//        = C - P(o+1) - Q(n-o),
// C = h[0] + the sum of every odd tap the filter reaches (offsets up to
// n-1 either way; it nearly cancels: formed in FP64 from the caller's taps),
// P(a) and Q(b) the sums of the odd taps at offsets >= a and <= -b (tails of
// small same-signed taps: FP32 suffix sums of the staged taps).  One extra
// warp forms C, P and Q while the others start their sums.
// Partial sums then stay near the size of the result (on a 2304 x 1472 fan
// sinogram: 1.3e-5 -> ~1e-6 from FP64).
#include <algorithm>

#include "ctr_common.cuh"

namespace ctr {
namespace {

constexpr int kWeightThreads = 256, kWeightWarps = kWeightThreads / 32;
constexpr int kWeightUnroll = 4;  // rows of a warp in flight
constexpr int kWeightCtas = 4;    // CTAs an SM, about

// The FP64 product w x rounded to float, as the reference rounds it, without
// FP64 arithmetic (its unit takes 16 cycles a warp's operation).  With w = wh +
// wl (both float) the product is p + t up to 2^-46 of it, p = x wh and t its
// remainder plus x wl, and r = p + t is its rounding to float unless the product
// lies that close to the midpoint of two floats: there, and outside the range
// where the remainders are exact, the product is formed in FP64.
__device__ __forceinline__ float weight_one(float x, float wh, float wl, double w)
{
    const float p = __fmul_rn(x, wh);
    const float t = __fmaf_rn(x, wl, __fmaf_rn(x, wh, -p));
    const float r = __fadd_rn(p, t);
    // what r leaves of p + t, and half a unit in r's last place
    const float d = fabsf(__fadd_rn(t, -__fadd_rn(r, -p)));
    const float half = __uint_as_float((__float_as_uint(r) & 0x7F800000u) - (24u << 23));
    const float a = fabsf(p);
    const bool fine = a > 1e-25f && a < 1e35f && fabsf(d - half) > half * 3.8e-6f && fabsf(d - 0.5f * half) > half * 3.8e-6f;
    if (fine) return r;
    if (x == 0.0f && fabsf(wh) < 1e35f) return p;  // with its sign
    return static_cast<float>(w * static_cast<double>(x));
}
__device__ __forceinline__ double weight_one(double x, float, float, double w) { return w * x; }

// A CTA weights 32 channels (a lane each) of a run of rows: one warp forms the
// FP64 weights, then every warp takes rows, a few in flight, each element read
// before it is written by the same thread (correct in place).  The launch has a
// few CTAs an SM, since each forms its weights anew: with 32-row CTAs of 128
// channels that took most of the time of a large batch.  16 x 1000 x 700: 95 ->
// 17.5 us (13 at the copy bandwidth); 2304 x 1472: 29 -> 7.6; 720 x 729: 6.5 ->
// 4.1; 180 x 185: 6.4 -> 3.3.  12 CTAs an SM: 23 us for the first.
template <typename T>
__global__ void __launch_bounds__(kWeightThreads)
    fan_weight_kernel(const T* in, T* out, unsigned ns, unsigned long long rows, unsigned long long per, double ds,
                      double cents, double dso, double dsd, int type)
{
    __shared__ double s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned is = blockIdx.x * 32 + lane;
    if (warp == 0) {
        const double s = ds * (static_cast<double>(is) - cents);
        s_w[lane] = type == 2 ? dso * fabs(cos(atan2(s, dsd))) / dsd : dso * fabs(cos(s / dsd)) / dsd;
    }
    __syncthreads();
    // launched as a dependent: the weights (kernel arguments only) are formed
    // while the kernel before it drains; global memory only after this wait
    grid_dep_wait();
    if (is >= ns) return;
    const double w = s_w[lane];
    const float wh = static_cast<float>(w), wl = static_cast<float>(w - static_cast<double>(wh));
    const unsigned long long r0 = blockIdx.y * per, r1 = rows - r0 < per ? rows : r0 + per;
    for (unsigned long long r = r0 + warp; r < r1; r += kWeightWarps * kWeightUnroll) {
        T v[kWeightUnroll];
#pragma unroll
        for (int i = 0; i < kWeightUnroll; ++i)
            v[i] = r + kWeightWarps * i < r1 ? in[(r + kWeightWarps * i) * ns + is] : T(0);
#pragma unroll
        for (int i = 0; i < kWeightUnroll; ++i)
            if (r + kWeightWarps * i < r1) out[(r + kWeightWarps * i) * ns + is] = weight_one(v[i], wh, wl, w);
    }
}

template <typename T>
int launch_fan_weighting(const ctr_fan_weighting_param* p, const T* in, T* out, int batch,
                         cudaStream_t stream)
{
    if (!p || bad_ptr(in) || bad_ptr(out)) return fail(CTR_ERR_INVALID_ARG, "null argument");
    int st = check_common(batch);
    if (st) return st;
    if (p->type != 1 && p->type != 2)
        return fail(CTR_ERR_INVALID_ARG, "fan weighting type %d (1 fan, 2 flat)", p->type);
    if (p->ns < 1 || p->nrow < 1) return fail(CTR_ERR_INVALID_ARG, "empty sinogram");
    const unsigned long long rows = static_cast<unsigned long long>(p->nrow) * batch;
    const double cents = static_cast<double>(p->ns - 1) / 2 + p->offset;
    if (div_up(rows, 32) > 65535u) return fail(CTR_ERR_UNSUPPORTED, "too many rows for one launch");
    // runs of whole passes of the CTA's warps, for about kWeightCtas CTAs an SM
    const unsigned columns = div_up(p->ns, 32);
    const unsigned long long step = kWeightWarps * kWeightUnroll;
    unsigned long long runs = std::max<unsigned long long>(1, static_cast<unsigned long long>(kWeightCtas) * device_sms() / columns);
    const unsigned long long per = std::max<unsigned long long>(1, (rows + runs * step - 1) / (runs * step)) * step;
    const cudaError_t e = launch_dependent(fan_weight_kernel<T>, dim3(columns, div_up(rows, per)), dim3(kWeightThreads), 0,
                                           stream, in, out, p->ns, rows, per, p->ds, cents, p->dso, p->dsd, p->type);
    if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "fan_weighting: %s", cudaGetErrorString(e));
    return check_launch("fan_weighting");
}

// ---- ramp filter ---------------------------------------------------------
//
// out[r][o] = ds * sum_j h[o - j] * x[r][j]   (correlation, the grad: h[j - o]).
// The ramp taps are zero at even offsets except 0, so output o sums the inputs
// of the other parity.  A thread computes 4 outputs of one parity, o_m = i0 + 2m,
// for kRows rows: stepping j by 2, the taps it needs, H[o_m - j], slide by one
// place (H[o_m - j - 2] = H[o_{m-1} - j]), so each step loads one new tap and
// one input per row for 4 * kRows FMAs, all from shared memory.  Thread pairs
// cover 8 consecutive outputs (both parities).  Even taps other than 0, which
// the ramp filters of the reference never have, take the generic loop.
constexpr int kFilterMaxThreads = 1024;
// Threads of the output tasks (the FP32 kernels add one warp, see filter_block).
constexpr int kFilterTaskThreads = kFilterMaxThreads - 32;
constexpr int kFilterPad = 16;   // zero taps beyond the ends of H
constexpr int kFilterRowsPlain = 2;
constexpr int kFilterRowsSpread = 3;

// Thread tasks of a row: (8-output block, parity).  When twice that fits one
// CTA, each task's inputs are split in two halves run by two threads, whose
// partial sums are added in a fixed order (halves the serial loop per thread).
__host__ __device__ inline int filter_tasks(unsigned ns) { return static_cast<int>((ns + 7) / 8) * 2; }
__host__ __device__ inline bool filter_split(unsigned ns) { return 2 * filter_tasks(ns) <= kFilterTaskThreads; }

__host__ __device__ inline int filter_threads(unsigned ns)
{
    const int t = filter_tasks(ns) * (filter_split(ns) ? 2 : 1);
    return t < 32 ? 32 : (t > kFilterTaskThreads ? kFilterTaskThreads : (t + 31) / 32 * 32);
}

// Tap storage: tap idx (offset d + ns - 1 + kFilterPad) lives at word
// tg*(idx/8) + idx%8.  With tg = 34 (skewed) a warp's lanes, which read taps
// i0 - j - 2 with i0 = 8q + p (q < 16, p < 2), fall in 32 distinct banks for
// every j; packed (tg = 8) the 16 groups of 8 fall in 8 banks (4-way
// conflicts).  The skewed layout is used where it fits the shared memory.
constexpr int kTapSkewed = 34, kTapPacked = 8;
__host__ __device__ inline int tap_slot(int idx, int tg) { return tg * (idx >> 3) + (idx & 7); }
__host__ __device__ inline int tap_words(unsigned ns, int tg)
{
    return tap_slot(2 * static_cast<int>(ns) + 2 * kFilterPad, tg);
}

// Shared layout (FP32): the tail sums P and Q of the odd taps [2][ns/2 + 2]
// and C (see filter_rows), then the taps H[-(ns-1) - kFilterPad .. ns - 1 +
// kFilterPad] (taps * ds), then xs[kRows][ns], then the second halves' sums
// [kRows][tasks][4].  FP64 has no tail sums.
__host__ __device__ inline size_t filter_tail_bytes(unsigned ns) { return (2 * (ns / 2 + 2) + 4) * sizeof(float); }
template <typename T>
__host__ __device__ inline size_t filter_smem(unsigned ns, int rows, int tg)
{
    return (sizeof(T) == 4 ? filter_tail_bytes(ns) : 0) +
           sizeof(T) * (static_cast<size_t>(tap_words(ns, tg)) + static_cast<size_t>(rows) * ns +
                        static_cast<size_t>(rows) * filter_tasks(ns) * 4);
}
// The FP32 kernels run one more warp, which forms C and the tail sums.
template <typename T>
__host__ __device__ inline int filter_block(unsigned ns)
{
    return filter_threads(ns) + (sizeof(T) == 4 ? 32 : 0);
}

// The tap layout for a launch: skewed when it fits kFilterSmemMax.
constexpr size_t kFilterSmemMax = 200 * 1024;
template <typename T>
inline int filter_layout(unsigned ns, int rows)
{
    return filter_smem<T>(ns, rows, kTapSkewed) <= kFilterSmemMax ? kTapSkewed : kTapPacked;
}

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// Inputs j = j0, j0 + 2, ... < j1 (one parity) into the four outputs i0, i0 + 2,
// i0 + 4, i0 + 6 of kRows rows; w0..w3 are the taps of input j0.  (Blocked
// partial sums cut the FP32 rounding of the long sums by ~1.3x on phantom
// sinograms and cost 11 % of the filter's time; not kept.)
template <typename T, int kRows>
__device__ __forceinline__ void filter_span(const T* __restrict__ xs, int n, int j0, int j1, int i0, int tg,
                                            const T* __restrict__ H0, T w0, T w1, T w2, T w3,
                                            const T (&cr)[kRows], T (&acc)[kRows][4])
{
    const int d0 = (n - 1) + kFilterPad;  // tap d sits at H0[tap_slot(d + d0, tg)]
#pragma unroll 4
    for (int j = j0; j < j1; j += 2) {
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const T xv = xs[r * n + j] - cr[r];
            acc[r][0] += w0 * xv;
            acc[r][1] += w1 * xv;
            acc[r][2] += w2 * xv;
            acc[r][3] += w3 * xv;
        }
        w3 = w2;
        w2 = w1;
        w1 = w0;
        w0 = H0[tap_slot(i0 - j - 2 + d0, tg)];
    }
}

template <typename T, int kRows, bool kGrad>
__device__ __forceinline__ void filter_rows(const T* __restrict__ in, const double* __restrict__ filter,
                                            T* __restrict__ out, const float* __restrict__ weight,
                                            unsigned ns, unsigned long long r0, int nr, double ds,
                                            int tg, unsigned char* smem_raw)
{
    constexpr bool kCentred = sizeof(T) == 4;
    const int n = static_cast<int>(ns);
    // FP32: the tail sums P [ns/2 + 2], Q [ns/2 + 2], then C
    const int nodd = n / 2;  // odd offsets in [1, n-1]
    float* Pt = reinterpret_cast<float*>(smem_raw);
    float* Qt = Pt + nodd + 2;
    float* Cs = Qt + nodd + 2;
    T* H0 = reinterpret_cast<T*>(smem_raw + (kCentred ? filter_tail_bytes(ns) : 0));
    const int d0 = (n - 1) + kFilterPad;  // tap d sits at H0[tap_slot(d + d0, tg)]
    auto H = [&](int d) -> T { return H0[tap_slot(d + d0, tg)]; };
    T* xs = H0 + tap_words(ns, tg);
    __shared__ int s_even;
    // the task threads; an FP32 block has one more warp (C and the tail sums)
    const int nthr = kCentred ? static_cast<int>(blockDim.x) - 32 : static_cast<int>(blockDim.x);

    const double* h = filter + ns;  // h[k], k in [-ns, ns]
    if (threadIdx.x == 0) s_even = 0;
    __syncthreads();
    {
        bool even = false;
        // staging loops unrolled so that a thread's global loads are in flight together
#pragma unroll 4
        for (int idx = threadIdx.x; idx < 2 * n + 2 * kFilterPad; idx += blockDim.x) {
            const int d = idx - (n - 1) - kFilterPad;
            double v = 0.0;
            if (d > -n && d < n) v = kGrad ? h[-d] : h[d];
            H0[tap_slot(idx, tg)] = static_cast<T>(v * ds);
            if (d != 0 && (d & 1) == 0 && v != 0.0) even = true;
        }
        if (even) s_even = 1;
#pragma unroll 4
        for (int idx = threadIdx.x; idx < kRows * n; idx += blockDim.x) {
            const int r = idx / n, j = idx - r * n;
            T v = 0;
            if (r < nr) {
                v = in[(r0 + r) * ns + j];
                if (weight) v = static_cast<T>(v * static_cast<T>(weight[j]));
            }
            xs[idx] = v;
        }
    }
    __syncthreads();
    if (kCentred && static_cast<int>(threadIdx.x) >= nthr) {
        // the extra warp, while the task threads start their sums.  Lanes 0-15
        // form P (positive offsets), lanes 16-31 Q (negative offsets): entry i
        // is the sum of the staged taps at odd offsets +-(2i+1) .. +-(n-1),
        // added from the far (small) end; entry nodd is 0.
        const int lane = threadIdx.x & 31, sl = lane & 15;
        const int sg = lane < 16 ? 1 : -1;
        float* A = lane < 16 ? Pt : Qt;
        const int C16 = (nodd + 15) / 16;
        const int i0 = min(sl * C16, nodd), i1 = min(i0 + C16, nodd);
        float tot = 0.0f;
        for (int i = i1 - 1; i >= i0; --i) tot += H(sg * (2 * i + 1));
        float suf = tot;  // inclusive suffix over this half's lanes
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
            const float v = __shfl_down_sync(0xffffffffu, suf, off, 16);
            if (sl + off < 16) suf += v;
        }
        suf -= tot;
        for (int i = i1 - 1; i >= i0; --i) {
            suf += H(sg * (2 * i + 1));
            A[i] = suf;
        }
        if (sl == 0) A[nodd] = A[nodd + 1] = 0.0f;
        // C in FP64 from the caller's taps
        double cs = 0.0;
        for (int i = lane; i < nodd; i += 32) {
            const int k = 2 * i + 1;
            cs += kGrad ? h[-k] + h[k] : h[k] + h[-k];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cs += __shfl_xor_sync(0xffffffffu, cs, off);
        if (lane == 0) Cs[0] = static_cast<float>((h[0] + cs) * ds);
    }
    // the single-thread-per-task path writes outputs as it goes: it needs the
    // sums first
    if (kCentred && !filter_split(ns)) __syncthreads();
    // D[o] (FP32 kernels), once per output
    auto dcorr = [&](int o) -> T {
        if constexpr (kCentred) return Cs[0] - Pt[(o + 1) / 2] - Qt[(n - o) / 2];
        else return T(0);
    };
    // output o of a thread whose reference value is c (FP32: centred sums)
    auto finish = [&](int o, int r, T c, T D, T acc) -> T {
        if constexpr (kCentred) return fma_t(H(0), xs[r * n + o] - c, fma_t(c, D, acc));
        else return fma_t(H(0), xs[r * n + o], acc);
    };
    // reference value of a task's rows: the input next to its outputs
    auto refs = [&](int i0, T (&cr)[kRows]) {
#pragma unroll
        for (int r = 0; r < kRows; ++r) cr[r] = kCentred ? xs[r * n + min(i0 + 3, n - 1)] : T(0);
    };
    const int groups = filter_tasks(ns);  // thread tasks: (8-output block, parity)
    T* red = xs + kRows * n;              // [kRows][groups][4]
    if (!s_even && filter_split(ns)) {
        // two threads per task (nthr >= 2 * groups): inputs [jb, jm) and [jm, n)
        const int task = threadIdx.x;
        const bool active = task < 2 * groups;
        const int half = task >= groups ? 1 : 0;
        const int g = task - half * groups;
        const int i0 = (g >> 1) * 8 + (g & 1);
        T acc[kRows][4], cr[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r)
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[r][m] = 0;
        if (active) {
            refs(i0, cr);
            const int jb = (i0 + 1) & 1;  // inputs of the other parity
            const int jm = jb + 2 * ((n - jb + 1) / 4);
            const int j0 = half ? jm : jb, j1 = half ? n : jm;
            T w0 = H(i0 - j0), w1 = H(i0 + 2 - j0), w2 = H(i0 + 4 - j0), w3 = H(i0 + 6 - j0);
            filter_span<T, kRows>(xs, n, j0, j1, i0, tg, H0, w0, w1, w2, w3, cr, acc);
            if (half) {
#pragma unroll
                for (int r = 0; r < kRows; ++r)
#pragma unroll
                    for (int m = 0; m < 4; ++m) red[(r * groups + g) * 4 + m] = acc[r][m];
            }
        }
        __syncthreads();
        if (active && !half) {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int o = i0 + 2 * m;
                if (o >= n) continue;
                const T D = dcorr(o);
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    if (r < nr)
                        out[(r0 + r) * ns + o] = finish(o, r, cr[r], D, acc[r][m] + red[(r * groups + g) * 4 + m]);
            }
        }
    } else if (!s_even) {
        for (int task = threadIdx.x; task < groups; task += blockDim.x) {
            const int i0 = (task >> 1) * 8 + (task & 1);
            T acc[kRows][4], cr[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int m = 0; m < 4; ++m) acc[r][m] = 0;
            refs(i0, cr);
            const int jb = (i0 + 1) & 1;  // inputs of the other parity
            T w0 = H(i0 - jb), w1 = H(i0 + 2 - jb), w2 = H(i0 + 4 - jb), w3 = H(i0 + 6 - jb);
            filter_span<T, kRows>(xs, n, jb, n, i0, tg, H0, w0, w1, w2, w3, cr, acc);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int o = i0 + 2 * m;
                if (o >= n) continue;
                const T D = dcorr(o);
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    if (r < nr) out[(r0 + r) * ns + o] = finish(o, r, cr[r], D, acc[r][m]);
            }
        }
    } else {
        // a filter with even taps: the plain sum over every input
        for (int o = threadIdx.x; o < n; o += blockDim.x) {
            T acc[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r) acc[r] = 0;
            for (int j = 0; j < n; ++j) {
                const T t = H(o - j);
#pragma unroll
                for (int r = 0; r < kRows; ++r) acc[r] += t * xs[r * n + j];
            }
#pragma unroll
            for (int r = 0; r < kRows; ++r)
                if (r < nr) out[(r0 + r) * ns + o] = acc[r];
        }
    }
    __syncthreads();  // shared buffers are free for the caller's next call
}

// ---- FP32, four rows at a time ------------------------------------------------
// filter_rows' sums for four rows as packed pairs and four outputs of a parity
// per thread.  The rows lie interleaved in shared memory, so an input of all
// four is one 16-byte load, and every tap is stored twice, so that it loads as
// the pair that multiplies two rows: a step is 2 loads, 2 packed differences and
// 8 packed multiply-adds for 16 products, where filter_span took 4 loads, 3
// differences and 12 multiply-adds for 12 (its loads bound it).  The inputs are
// split over groups of threads, whose sums are added in order; how, depends on
// the channels alone, so that a row's result does not on the rows beside it.
// Bound by the packed FP32 unit, 10 operations a step.  720 x 729: 24.3 -> 23.7
// us; 4 x 720 x 729: 84 -> 52; 16 x 1000 x 700: 392 -> 248; 2304 x 1472: 238 -> 147;
// 1472 x 2304: 381 -> 285.  Eight outputs a thread with one reference value took
// 20.9, 48, 207, 149 and 333, and cost digits (phantoms on 500 channels 5.9e-7 from
// FP64 in filter_rows, 9.3e-7 so, here 4.5e-7); with two reference values they
// spill (255 us for the third).
constexpr int kQuadRows = 4, kQuadOut = 4;
constexpr size_t kQuadSmemMax = 226 * 1024;
constexpr int kQuadThreads = 384;  // task threads of a CTA, two CTAs an SM
constexpr int kQuadWide = 992;     // those of rows with more tasks, where they fit
// Tap idx lies at pair 10 (idx / 8) + idx % 8: the 16 lanes of a half-warp's
// load (taps 8 q + p, q < 8, p < 2) fall in distinct banks.
constexpr int kQuadGroup = 10;
__host__ __device__ inline int quad_slot(int idx) { return kQuadGroup * (idx >> 3) + (idx & 7); }
__host__ __device__ inline int quad_taps(unsigned ns) { return quad_slot(2 * static_cast<int>(ns) + 2 * kFilterPad + 8); }
// Tasks (filter_tasks: 8-output block, parity) of a row and the parts that their
// inputs are split into, each rounded up to whole warps; one more warp forms C and
// the tail sums.
__host__ __device__ inline int quad_stride(unsigned ns) { return (filter_tasks(ns) + 31) / 32 * 32; }
__host__ __device__ inline int quad_parts(unsigned ns)
{
    const int p = kQuadThreads / quad_stride(ns);
    return p < 1 ? 1 : (p > 8 ? 8 : p);
}
inline int quad_block(unsigned ns, int threads)
{
    const int t = quad_stride(ns);
    return (t > threads ? threads : t * quad_parts(ns)) + 32;
}
// A thread's sums are put by in shared memory at least every kQuadFold inputs
// (blocked summation), where there is room for it: 1472 channels 2.0e-6 from FP64
// in one sum of 736, 7.9e-7 in two halves, 4.7e-7 so.
constexpr int kQuadFold = 128;
constexpr unsigned kFilterBatchMaxNs = 4904;  // of a batched launch
// Threads that take tasks: the extra warp too, once the tasks are more than a CTA's.
inline int quad_slots(unsigned ns, int nthr) { return filter_tasks(ns) > nthr ? nthr + 32 : nthr; }
// Shared layout: inputs [ns] of four rows, the threads' sums [output][slot], taps,
// tail sums.
inline size_t quad_smem(unsigned ns, int slots)
{
    return sizeof(float4) * (ns + kQuadOut * slots) + sizeof(float2) * quad_taps(ns) + filter_tail_bytes(ns);
}

__device__ __forceinline__ float2 pair_of(float v) { return make_float2(v, v); }

// Inputs j0, j0 + 2, ... < j1, less the reference values c, into the outputs
// i0 + 2 m: acc[m][0] rows 0 and 1, acc[m][1] rows 2 and 3.
__device__ __forceinline__ void quad_span(const float4* __restrict__ xs, int j0, int j1, int i0, int d0,
                                          const float2* __restrict__ Hd, const float4& c,
                                          float2 (&acc)[kQuadOut][2])
{
    const float2 minus = pair_of(-1.0f);
    int idx = i0 - j0 + d0;  // the tap of output i0 and input j
    float2 w[kQuadOut];      // tap of output m at w[(m - turn) % 4]
#pragma unroll
    for (int m = 0; m < kQuadOut; ++m) w[m] = Hd[quad_slot(idx + 2 * m)];
    // eight inputs move the taps by two groups: the same places twenty pairs back
    const float2* h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = Hd + quad_slot(idx - 2 - 2 * k);
    int j = j0;
    auto step = [&](float4 x, int turn) {
        const float2 xa = __ffma2_rn(make_float2(c.x, c.y), minus, make_float2(x.x, x.y));
        const float2 xb = __ffma2_rn(make_float2(c.z, c.w), minus, make_float2(x.z, x.w));
#pragma unroll
        for (int m = 0; m < kQuadOut; ++m) {
            acc[m][0] = __ffma2_rn(w[(m + 2 * kQuadOut - turn) % kQuadOut], xa, acc[m][0]);
            acc[m][1] = __ffma2_rn(w[(m + 2 * kQuadOut - turn) % kQuadOut], xb, acc[m][1]);
        }
    };
    for (; j + 14 < j1; j += 16) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            step(xs[j + 2 * k], k);
            w[(7 - k) % kQuadOut] = h[k & 3][k < 4 ? 0 : -kQuadGroup];  // the new tap takes the place of the last output's
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] -= 2 * kQuadGroup;
        idx -= 16;
    }
    for (; j < j1; j += 2) {
        step(xs[j], 0);
#pragma unroll
        for (int m = kQuadOut - 1; m > 0; --m) w[m] = w[m - 1];
        idx -= 2;
        w[0] = Hd[quad_slot(idx)];
    }
}

template <bool kGrad>
__device__ __forceinline__ void filter_quad(const float* __restrict__ in, const double* __restrict__ filter,
                                            float* __restrict__ out, const float* __restrict__ weight, unsigned ns,
                                            unsigned long long r0, int nr, double ds, int slots,
                                            unsigned char* smem_raw)
{
    const int n = static_cast<int>(ns), nodd = n / 2;  // odd offsets in [1, n-1]
    const int tasks = filter_tasks(ns);
    float4* xs = reinterpret_cast<float4*>(smem_raw);
    const int nthr = static_cast<int>(blockDim.x) - 32;  // the task threads; one more warp forms C and the tail sums
    const int parts = quad_parts(ns);
    float4* red = xs + n;  // [output][thread]
    float2* Hd = reinterpret_cast<float2*>(red + kQuadOut * slots);
    float* Pt = reinterpret_cast<float*>(Hd + quad_taps(ns));
    float* Qt = Pt + nodd + 2;
    float* Cs = Qt + nodd + 2;
    const int d0 = (n - 1) + kFilterPad;
    auto H = [&](int d) { return Hd[quad_slot(d + d0)].x; };
    __shared__ int s_even;

    const double* h = filter + ns;  // h[k], k in [-ns, ns]
    if (threadIdx.x == 0) s_even = 0;
    __syncthreads();
    {
        bool even = false;
#pragma unroll 4
        for (int idx = threadIdx.x; idx < 2 * n + 2 * kFilterPad; idx += blockDim.x) {
            const int d = idx - (n - 1) - kFilterPad;
            double v = 0.0;
            if (d > -n && d < n) v = kGrad ? h[-d] : h[d];
            // zeros (every even tap but 0 of the reference's filters) without FP64 arithmetic
            const bool zero = (__double_as_longlong(v) << 1) == 0;
            Hd[quad_slot(idx)] = pair_of(zero ? 0.0f : static_cast<float>(v * ds));
            if (d != 0 && (d & 1) == 0 && !zero) even = true;
        }
        if (even) s_even = 1;
        const float* row = in + r0 * ns;
#pragma unroll 2
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            float4 v = make_float4(row[j], nr > 1 ? row[ns + j] : 0.0f, nr > 2 ? row[2 * static_cast<size_t>(ns) + j] : 0.0f,
                                   nr > 3 ? row[3 * static_cast<size_t>(ns) + j] : 0.0f);
            if (weight) {
                const float w = weight[j];
                v = make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
            }
            xs[j] = v;
        }
    }
    __syncthreads();
    if (static_cast<int>(threadIdx.x) >= nthr) {  // as in filter_rows
        const int lane = threadIdx.x & 31, sl = lane & 15;
        const int sg = lane < 16 ? 1 : -1;
        float* A = lane < 16 ? Pt : Qt;
        const int C16 = (nodd + 15) / 16;
        const int i0 = min(sl * C16, nodd), i1 = min(i0 + C16, nodd);
        float tot = 0.0f;
        for (int i = i1 - 1; i >= i0; --i) tot += H(sg * (2 * i + 1));
        float suf = tot;
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
            const float v = __shfl_down_sync(0xffffffffu, suf, off, 16);
            if (sl + off < 16) suf += v;
        }
        suf -= tot;
        for (int i = i1 - 1; i >= i0; --i) {
            suf += H(sg * (2 * i + 1));
            A[i] = suf;
        }
        if (sl == 0) A[nodd] = A[nodd + 1] = 0.0f;
        double cs = 0.0;
#pragma unroll 8
        for (int i = lane; i < nodd; i += 32) {  // the loads in flight together
            const int k = 2 * i + 1;
            cs += kGrad ? h[-k] + h[k] : h[k] + h[-k];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cs += __shfl_xor_sync(0xffffffffu, cs, off);
        if (lane == 0) Cs[0] = static_cast<float>((h[0] + cs) * ds);
    }
    if (parts == 1) __syncthreads();  // the tasks write outputs as they go: the sums first
    // the reference value of a task's rows: the input next to its outputs
    auto refs = [&](int i0) { return xs[min(i0 + 3, n - 1)]; };
    // this thread's sums over the inputs ja, ja + 2, ... < je, at most kQuadFold at a
    // time, the earlier ones' total in `red`
    auto sums = [&](int ja, int je, int i0, const float4& c, float2 (&acc)[kQuadOut][2]) {
        const int cnt = (je - ja + 1) / 2, folds = slots > 0 ? max(1, (cnt + kQuadFold - 1) / kQuadFold) : 1;
        float4* own = red + threadIdx.x;
        for (int k = 0; k < folds; ++k) {
#pragma unroll
            for (int m = 0; m < kQuadOut; ++m) acc[m][0] = acc[m][1] = make_float2(0.0f, 0.0f);
            quad_span(xs, ja + 2 * (cnt * k / folds), k + 1 == folds ? je : ja + 2 * (cnt * (k + 1) / folds), i0, d0, Hd, c, acc);
            if (folds == 1) return;
#pragma unroll
            for (int m = 0; m < kQuadOut; ++m) {
                if (k > 0) {
                    const float4 v = own[m * slots];
                    acc[m][0] = __fadd2_rn(acc[m][0], make_float2(v.x, v.y));
                    acc[m][1] = __fadd2_rn(acc[m][1], make_float2(v.z, v.w));
                }
                if (k + 1 < folds) own[m * slots] = make_float4(acc[m][0].x, acc[m][0].y, acc[m][1].x, acc[m][1].y);
            }
        }
    };
    // outputs i0, i0 + 2, ... of a task
    auto finish = [&](int i0, const float4& c, const float2 (&acc)[kQuadOut][2]) {
        const float h0 = H(0);
#pragma unroll
        for (int m = 0; m < kQuadOut; ++m) {
            const int o = i0 + 2 * m;
            if (o >= n) continue;
            const float D = Cs[0] - Pt[(o + 1) / 2] - Qt[(n - o) / 2];
            const float4 x = xs[o];
            float* to = out + r0 * ns + o;
            to[0] = fmaf(h0, x.x - c.x, fmaf(c.x, D, acc[m][0].x));
            if (nr > 1) to[ns] = fmaf(h0, x.y - c.y, fmaf(c.y, D, acc[m][0].y));
            if (nr > 2) to[2 * static_cast<size_t>(ns)] = fmaf(h0, x.z - c.z, fmaf(c.z, D, acc[m][1].x));
            if (nr > 3) to[3 * static_cast<size_t>(ns)] = fmaf(h0, x.w - c.w, fmaf(c.w, D, acc[m][1].y));
        }
    };
    if (!s_even && parts > 1) {
        const int stride = quad_stride(ns), part = threadIdx.x / stride, g = threadIdx.x - part * stride;
        const bool active = part < parts && g < tasks;
        const int i0 = (g >> 1) * 8 + (g & 1);
        float2 acc[kQuadOut][2] = {};
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (active) {
            c = refs(i0);
            const int jb = (i0 + 1) & 1;  // inputs of the other parity
            const int cnt = (n - jb + 1) / 2;
            sums(jb + 2 * (cnt * part / parts), part + 1 == parts ? n : jb + 2 * (cnt * (part + 1) / parts), i0, c, acc);
            if (part > 0) {
#pragma unroll
                for (int m = 0; m < kQuadOut; ++m)
                    red[m * slots + threadIdx.x] = make_float4(acc[m][0].x, acc[m][0].y, acc[m][1].x, acc[m][1].y);
            }
        }
        __syncthreads();
        if (active && part == 0) {
            for (int k = 1; k < parts; ++k)
#pragma unroll
                for (int m = 0; m < kQuadOut; ++m) {
                    const float4 v = red[m * slots + k * stride + g];
                    acc[m][0] = __fadd2_rn(acc[m][0], make_float2(v.x, v.y));
                    acc[m][1] = __fadd2_rn(acc[m][1], make_float2(v.z, v.w));
                }
            finish(i0, c, acc);
        }
    } else if (!s_even) {
        for (int task = threadIdx.x; task < tasks; task += blockDim.x) {
            const int i0 = (task >> 1) * 8 + (task & 1);
            float2 acc[kQuadOut][2];
            const float4 c = refs(i0);
            sums((i0 + 1) & 1, n, i0, c, acc);
            finish(i0, c, acc);
        }
    } else {
        // a filter with even taps: the plain sum over every input
        for (int o = threadIdx.x; o < n; o += blockDim.x) {
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int j = 0; j < n; ++j) {
                const float t = H(o - j);
                const float4 x = xs[j];
                a = make_float4(fmaf(t, x.x, a.x), fmaf(t, x.y, a.y), fmaf(t, x.z, a.z), fmaf(t, x.w, a.w));
            }
            float* to = out + r0 * ns + o;
            to[0] = a.x;
            if (nr > 1) to[ns] = a.y;
            if (nr > 2) to[2 * static_cast<size_t>(ns)] = a.z;
            if (nr > 3) to[3 * static_cast<size_t>(ns)] = a.w;
        }
    }
}

template <bool kGrad, int kThreads, int kCtas>
__global__ void __launch_bounds__(kThreads + 32, kCtas)
    ramp_filter_quad(const float* __restrict__ in, const double* __restrict__ filter, float* __restrict__ out,
                     const float* __restrict__ weight, unsigned ns, unsigned long long rows, double ds, int slots)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    grid_dep_wait();  // launched as a dependent of the kernel before it
    // rows dealt evenly over the grid, at most kQuadRows a CTA
    const unsigned long long r0 = blockIdx.x * rows / gridDim.x, r1 = (blockIdx.x + 1ull) * rows / gridDim.x;
    filter_quad<kGrad>(in, filter, out, weight, ns, r0, static_cast<int>(r1 - r0), ds, slots, smem_raw);
}

// False (nothing launched) where a row does not fit the shared memory.
template <bool kGrad, int kThreads, int kCtas>
bool launch_quad(const ctr_filter_param* p, const float* in, const double* filter, float* out, const float* weight,
                 unsigned long long rows, cudaStream_t stream, cudaError_t* e)
{
    const int block = quad_block(p->ns, kThreads);
    int slots = quad_slots(p->ns, block - 32);
    if (kThreads == kQuadWide && quad_smem(p->ns, slots) > kQuadSmemMax) slots = 0;  // one sum a thread
    const size_t smem = quad_smem(p->ns, slots);
    const unsigned long long blocks = (rows + kQuadRows - 1) / kQuadRows;
    auto kern = ramp_filter_quad<kGrad, kThreads, kCtas>;
    if (smem > kQuadSmemMax || blocks > 0x7fffffffull ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    *e = launch_dependent(kern, dim3(static_cast<unsigned>(blocks)), dim3(block), smem, stream, in,
                          filter, out, weight, p->ns, rows, p->ds, slots);
    return true;
}

// kRows rows a CTA; with `spread` the rows are instead dealt evenly over the
// grid (CTA i: rows [i*rows/G, (i+1)*rows/G), at most kRows), so a grid of
// exactly the resident CTAs finishes in one wave.
template <typename T, bool kGrad, int kRows>
__global__ void __launch_bounds__(kFilterMaxThreads)
    ramp_filter_kernel(const T* __restrict__ in, const double* __restrict__ filter,
                       T* __restrict__ out, const float* __restrict__ weight, unsigned ns,
                       unsigned long long rows, double ds, int tg, int spread)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    grid_dep_wait();  // launched as a dependent of the kernel before it
    unsigned long long r0, r1;
    if (spread) {
        r0 = static_cast<unsigned long long>(blockIdx.x) * rows / gridDim.x;
        r1 = static_cast<unsigned long long>(blockIdx.x + 1) * rows / gridDim.x;
    } else {
        r0 = static_cast<unsigned long long>(blockIdx.x) * kRows;
        r1 = rows - r0 < kRows ? rows : r0 + kRows;
    }
    filter_rows<T, kRows, kGrad>(in, filter, out, weight, ns, r0, static_cast<int>(r1 - r0), ds, tg, smem_raw);
}

// Batched FP32 filtering with pre-weighting: one CTA per (job, row block).
__global__ void __launch_bounds__(kQuadThreads + 32, 2)
    ramp_filter_batch_kernel(const FilterJob* __restrict__ jobs, const int2* __restrict__ blocks, int slots)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int2 b = blocks[blockIdx.x];  // (job, first row)
    const FilterJob J = jobs[b.x];
    const int nr = min(kFilterRowsPerBlock, static_cast<int>(J.nrow) - b.y);
    static_assert(kFilterRowsPerBlock == kQuadRows, "a block's rows");
    filter_quad<false>(J.in, J.taps, J.out, J.weight, J.ns, b.y, nr, J.ds, slots, smem_raw);
}

template <typename T, bool kGrad>
int launch_ramp_filter(const ctr_filter_param* p, const T* in, const double* filter, T* out,
                       const float* weight, int batch, cudaStream_t stream)
{
    if (!p || bad_ptr(in) || bad_ptr(filter) || bad_ptr(out))
        return fail(CTR_ERR_INVALID_ARG, "null argument");
    int st = check_common(batch);
    if (st) return st;
    if (p->ns < 1 || p->nrow < 1) return fail(CTR_ERR_INVALID_ARG, "empty sinogram");
    if (in == out) return fail(CTR_ERR_INVALID_ARG, "ramp filter cannot run in place");
    const unsigned long long rows = static_cast<unsigned long long>(p->nrow) * batch;
    const int threads = filter_block<T>(p->ns);
    if constexpr (sizeof(T) == 4) {
        cudaError_t e = cudaSuccess;
        if (quad_stride(p->ns) > kQuadThreads ? launch_quad<kGrad, kQuadWide, 1>(p, in, filter, out, weight, rows, stream, &e)
                                              : launch_quad<kGrad, kQuadThreads, 2>(p, in, filter, out, weight, rows, stream, &e)) {
            if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "ramp_filter: %s", cudaGetErrorString(e));
            return check_launch("ramp_filter");
        }
    }
    // Up to kFilterRowsSpread rows a CTA dealt over the resident CTAs (one
    // wave, CTAs within a row of each other); more rows take CTAs of
    // kFilterRowsPlain rows in waves.
    {
        const int tg = filter_layout<T>(p->ns, kFilterRowsSpread);
        const size_t smem = filter_smem<T>(p->ns, kFilterRowsSpread, tg);
        auto kern = ramp_filter_kernel<T, kGrad, kFilterRowsSpread>;
        int per_sm = 0;
        if (smem <= kFilterSmemMax &&
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) ==
                cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) == cudaSuccess &&
            per_sm > 0) {
            const unsigned long long resident = static_cast<unsigned long long>(per_sm) * device_sms();
            if (rows <= kFilterRowsSpread * resident) {
                const unsigned blocks = static_cast<unsigned>(rows < resident ? rows : resident);
                const cudaError_t e = launch_dependent(kern, dim3(blocks), dim3(threads), smem, stream, in, filter,
                                                       out, weight, p->ns, rows, p->ds, tg, 1);
                if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "ramp_filter: %s", cudaGetErrorString(e));
                return check_launch("ramp_filter");
            }
        }
        cudaGetLastError();
    }
    const int tg = filter_layout<T>(p->ns, kFilterRowsPlain);
    const size_t smem = filter_smem<T>(p->ns, kFilterRowsPlain, tg);
    if (smem > kFilterSmemMax)
        return fail(CTR_ERR_UNSUPPORTED, "ns=%u exceeds the filter's shared-memory tile", p->ns);
    auto kern = ramp_filter_kernel<T, kGrad, kFilterRowsPlain>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "filter smem: %s", cudaGetErrorString(e));
    const unsigned blocks = div_up(rows, kFilterRowsPlain);
    e = launch_dependent(kern, dim3(blocks), dim3(threads), smem, stream, in, filter, out, weight, p->ns, rows,
                         p->ds, tg, 0);
    if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "ramp_filter: %s", cudaGetErrorString(e));
    return check_launch("ramp_filter");
}

}  // namespace

int ramp_filter_weighted_f32(const ctr_filter_param* p, const float* in, const double* filter,
                             float* out, const float* weight, int batch, cudaStream_t stream)
{
    return launch_ramp_filter<float, false>(p, in, filter, out, weight, batch, stream);
}

// Batched weighting + filtering of a job list (see FilterJob); `blocks` lists
// (job, first row) pairs, one CTA each; max_ns sizes the shared memory.
int ramp_filter_batch_f32(const FilterJob* jobs, const int2* blocks, int n_blocks, unsigned max_ns,
                          cudaStream_t stream)
{
    const int slots = quad_slots(max_ns, kQuadThreads);
    const size_t smem = quad_smem(max_ns, slots);
    if (max_ns > kFilterBatchMaxNs) return fail(CTR_ERR_UNSUPPORTED, "ns=%u too wide for the filter tile", max_ns);
    cudaError_t e = cudaFuncSetAttribute(ramp_filter_batch_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return fail(CTR_ERR_CUDA, "filter smem: %s", cudaGetErrorString(e));
    if (n_blocks > 0) ramp_filter_batch_kernel<<<n_blocks, kQuadThreads + 32, smem, stream>>>(jobs, blocks, slots);
    return check_launch("ramp_filter_batch");
}

}  // namespace ctr

using namespace ctr;

extern "C" {

int ctr_fan_weighting_f32(const ctr_fan_weighting_param* p, const float* in, float* out,
                          int batch, cudaStream_t stream)
{
    return launch_fan_weighting<float>(p, in, out, batch, stream);
}
int ctr_fan_weighting_f64(const ctr_fan_weighting_param* p, const double* in, double* out,
                          int batch, cudaStream_t stream)
{
    return launch_fan_weighting<double>(p, in, out, batch, stream);
}
// The reference's grad applies the same diagonal weight (src/fan_weighting.cc:40-59).
int ctr_fan_weighting_grad_f32(const ctr_fan_weighting_param* p, const float* in, float* out,
                               int batch, cudaStream_t stream)
{
    return launch_fan_weighting<float>(p, in, out, batch, stream);
}
int ctr_fan_weighting_grad_f64(const ctr_fan_weighting_param* p, const double* in,
                               double* out, int batch, cudaStream_t stream)
{
    return launch_fan_weighting<double>(p, in, out, batch, stream);
}

int ctr_ramp_filter_f32(const ctr_filter_param* p, const float* in, const double* filter,
                        float* out, int batch, cudaStream_t stream)
{
    return launch_ramp_filter<float, false>(p, in, filter, out, nullptr, batch, stream);
}
int ctr_ramp_filter_f64(const ctr_filter_param* p, const double* in, const double* filter,
                        double* out, int batch, cudaStream_t stream)
{
    return launch_ramp_filter<double, false>(p, in, filter, out, nullptr, batch, stream);
}
int ctr_ramp_filter_grad_f32(const ctr_filter_param* p, const float* in, const double* filter,
                             float* out, int batch, cudaStream_t stream)
{
    return launch_ramp_filter<float, true>(p, in, filter, out, nullptr, batch, stream);
}
int ctr_ramp_filter_grad_f64(const ctr_filter_param* p, const double* in,
                             const double* filter, double* out, int batch,
                             cudaStream_t stream)
{
    return launch_ramp_filter<double, true>(p, in, filter, out, nullptr, batch, stream);
}

}  // extern "C"
