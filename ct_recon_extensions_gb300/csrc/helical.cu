// Helical rebinning: 3-D helical sinograms to 2-D fan-beam sinograms, one per
// reconstructed slice, by 360LI or 180LI z interpolation (reference
// src/helical_interpolation.cc:80-370, include/helical_interpolation.h).
//
// The reference runs this on the CPU only.  Here one thread computes one
// output sample (slice, view, channel).  T=double runs the exact kernel: every
// operation is an FP64 intrinsic in the reference's order (__dadd_rn and
// friends, so nothing is contracted into an FMA), and the per-channel
// cos(gamma) and per-slice view ranges come from the host
// (ctr_helical_interpolation_prep) with the reference's own libm calls, so the
// output equals the reference's bit for bit.  T=float runs the FP32 fast path
// (helical_360_f32, helical_fast_f32): the same decisions as the reference (rows, usability,
// views) with FP32 sums, falling back to the exact computation per sample
// where an FP32 decision could differ; GB300's FP64 rate is 1/64 of its FP32
// rate, which made the exact kernel compute-bound at <1 % of HBM bandwidth.
//
// Layout: input [na][nt][ns] (view, detector row, channel), output
// [nz][view_per_rot][ns]; a block covers 128 consecutive channels of one
// (slice, view) row, so every row read is a coalesced channel run.
#include <cmath>
#include <type_traits>
#include <vector>

#include "ctr_common.cuh"

namespace ctr {
namespace {

constexpr int kHeliThreads = 128;
constexpr double kHeliPi = 3.14159265358979323846;  // M_PI of the reference's <cmath>

// Device table written by ctr_helical_interpolation_prep: a header, then one
// HeliChan per channel, then one HeliSlice per slice.
struct HeliHeader {
    int method;  // CTR_HELICAL_360 or CTR_HELICAL_180
    unsigned ns, nz, vpr;
};
struct HeliChan {
    double cg;    // cos(gamma), gamma = (is - center_s) * ds / dsd
    double dif;   // 180LI: views back to the complementary ray, (pi - 2 gamma) / orbit
    double sc;    // 180LI: the complementary ray's channel, center_s - s / ds
    double pad;
};
struct HeliSlice {
    double z;                   // slice position, z0 + dz added iz times
    int center, lo, hi, first;  // nearest view, view range [lo, hi], first output view
    int valid;                  // 0: [lo, hi] leaves the scan ("View not enough for this slice!")
    int pad;
};
static_assert(sizeof(HeliHeader) == 16 && sizeof(HeliChan) == 32 && sizeof(HeliSlice) == 32,
              "table layout");

struct HeliGeo {
    unsigned ns, nt, na, vpr, nz;
    double center_t, couch_begin, couch_mov, half_th, dso, dsd, nt_d, ns_last;
    size_t in_item, out_item;
    float ct_f, nt_f, hth_f, vprcm_f;  // FP32 fast path: center_t, nt, thickness / 2, vpr * couch_mov
};

// Rows [r0, r1) the thick slice covers for a source z_dif below the slice:
// the slab edges projected onto the detector, clamped to it
// (src/helical_interpolation.cc:105-111).  false when the slab misses.
__device__ __forceinline__ bool heli_rows(const HeliGeo& g, double zd, double cg, int& r0, int& r1)
{
    const double top = __dsub_rn(g.center_t,
                                 __dmul_rn(__dmul_rn(__ddiv_rn(__dadd_rn(zd, g.half_th), g.dso), cg), g.dsd));
    const double bot = __dsub_rn(g.center_t,
                                 __dmul_rn(__dmul_rn(__ddiv_rn(__dsub_rn(zd, g.half_th), g.dso), cg), g.dsd));
    if (bot < 0.0 || top >= g.nt_d) return false;
    r0 = static_cast<int>(floor(top < 0.0 ? 0.0 : top));
    r1 = static_cast<int>(ceil(bot >= g.nt_d ? g.nt_d : bot));
    return true;
}

// Rows in [r0, r1): the reference's loop count (0 for an inverted slab, so
// that its mean is 0/0 as there).
__device__ __forceinline__ double heli_count(int r0, int r1) { return static_cast<double>(r1 > r0 ? r1 - r0 : 0); }

// Mean over rows [r0, r1) of one channel column (stride ns between rows).
template <typename T>
__device__ __forceinline__ double heli_mean(const T* __restrict__ col, unsigned ns, int r0, int r1)
{
    double acc = 0.0;
    for (int r = r0; r < r1; ++r)
        acc = __dadd_rn(acc, static_cast<double>(__ldg(col + static_cast<size_t>(r) * ns)));
    return __ddiv_rn(acc, heli_count(r0, r1));
}

// One sample of a 180LI complementary ray; views outside [0, na) read as 0
// and raise CTR_HELICAL_OUTSIDE (the reference indexes out of bounds there).
template <typename T>
__device__ __forceinline__ double heli_at(const T* __restrict__ in, const HeliGeo& g, int view, int r, int c,
                                          bool& outside)
{
    if (view < 0 || static_cast<unsigned>(view) >= g.na) {
        outside = true;
        return 0.0;
    }
    return static_cast<double>(__ldg(in + (static_cast<size_t>(view) * g.nt + r) * g.ns + c));
}

// The reference's value of one output sample (slice s, output view iv,
// channel is), in FP64 and bit for bit: src/helical_interpolation.cc:93-149
// (360LI) and 169-248 (180LI).  ORs CTR_HELICAL_NO_ROWS / _OUTSIDE into *status.
template <typename T, int M>
__device__ double heli_exact(const T* __restrict__ in, const HeliGeo& g, const HeliSlice& s, const HeliChan& c,
                             unsigned iv, unsigned is, unsigned* status)
{
    const size_t view_stride = static_cast<size_t>(g.nt) * g.ns;
    const double zrel = __dsub_rn(s.z, g.couch_begin);  // z - couch_begin, then - view * couch_mov
    int cur = s.first + static_cast<int>(iv);
    if (M == CTR_HELICAL_180 && cur > s.hi) cur -= static_cast<int>(g.vpr);
    const double zd = __dsub_rn(zrel, __dmul_rn(static_cast<double>(cur), g.couch_mov));

    int r0 = 0, r1 = 0;
    double vcur = 0.0, vcor = 0.0, zd2;
    const bool ucur = heli_rows(g, zd, c.cg, r0, r1);
    if (ucur) vcur = heli_mean(in + cur * view_stride + is, g.ns, r0, r1);

    bool ucor;
    if (M == CTR_HELICAL_360) {
        // the view one rotation away, on the other side of the slice
        const int cor = cur >= s.center ? cur - static_cast<int>(g.vpr) : cur + static_cast<int>(g.vpr);
        zd2 = __dsub_rn(zrel, __dmul_rn(static_cast<double>(cor), g.couch_mov));
        ucor = heli_rows(g, zd2, c.cg, r0, r1);
        if (ucor) vcor = heli_mean(in + cor * view_stride + is, g.ns, r0, r1);
    } else {
        // the complementary ray: (pi - 2 gamma) / orbit views back, wrapped into [lo, hi] once each way
        double cv = __dsub_rn(static_cast<double>(cur), c.dif);
        if (cv < static_cast<double>(s.lo)) cv = __dadd_rn(cv, static_cast<double>(g.vpr));
        if (cv > static_cast<double>(s.hi)) cv = __dsub_rn(cv, static_cast<double>(g.vpr));
        zd2 = __dsub_rn(zrel, __dmul_rn(cv, g.couch_mov));
        ucor = heli_rows(g, zd2, c.cg, r0, r1);
        if (ucor) {
            const int vl = static_cast<int>(floor(cv)), vr = static_cast<int>(ceil(cv));
            const double u = __dsub_rn(cv, static_cast<double>(vl));
            if (c.sc < 0.0 || c.sc > g.ns_last) return vcur;  // mirrored channel off the detector
            const int cl = static_cast<int>(floor(c.sc)), cr = static_cast<int>(ceil(c.sc));
            const double v = __dsub_rn(c.sc, static_cast<double>(cl)), w = __dsub_rn(1.0, v);
            double left = 0.0, right = 0.0;
            bool outside = false;
            for (int r = r0; r < r1; ++r) {
                left = __dadd_rn(left, __dadd_rn(__dmul_rn(w, heli_at(in, g, vl, r, cl, outside)),
                                                 __dmul_rn(v, heli_at(in, g, vl, r, cr, outside))));
                right = __dadd_rn(right, __dadd_rn(__dmul_rn(w, heli_at(in, g, vr, r, cl, outside)),
                                                   __dmul_rn(v, heli_at(in, g, vr, r, cr, outside))));
            }
            if (outside) atomicOr(status, CTR_HELICAL_OUTSIDE);
            vcor = __ddiv_rn(__dadd_rn(__dmul_rn(__dsub_rn(1.0, u), left), __dmul_rn(u, right)),
                             heli_count(r0, r1));
        }
    }
    if (ucur && ucor) return __ddiv_rn(__dsub_rn(__dmul_rn(zd, vcor), __dmul_rn(zd2, vcur)), __dsub_rn(zd, zd2));
    if (ucur) return vcur;
    if (ucor) return vcor;
    atomicOr(status, CTR_HELICAL_NO_ROWS);  // the reference throws "No row data available!"
    return 0.0;
}

// Table checks shared by both kernels: false (and nothing to do) for a table
// of another method or geometry, or for a slice the reference rejects.
template <int M>
__device__ __forceinline__ bool heli_slice_ok(const HeliHeader* tab, const HeliGeo& g, const HeliSlice& s,
                                              unsigned* status)
{
    if (tab->method != M || tab->ns != g.ns || tab->nz != g.nz || tab->vpr != g.vpr) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
            atomicOr(status, CTR_HELICAL_BAD_TABLE);
        return false;
    }
    if (!s.valid) {  // the reference throws before touching this slice
        if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) atomicOr(status + blockIdx.z, CTR_HELICAL_NO_VIEWS);
        return false;
    }
    return true;
}

template <int M>
__device__ __forceinline__ const HeliSlice* heli_slices(const HeliHeader* tab, const HeliGeo& g)
{
    return reinterpret_cast<const HeliSlice*>(reinterpret_cast<const HeliChan*>(tab + 1) + g.ns);
}

// The exact kernel (T=double, and T=float where the fast path's conditions do
// not hold): every sample through heli_exact.
template <typename T, int M>
__global__ void __launch_bounds__(kHeliThreads)
    helical_kernel(const T* __restrict__ in, T* __restrict__ out, const HeliHeader* __restrict__ tab, HeliGeo g,
                   unsigned* status)
{
    const unsigned iz = blockIdx.z % g.nz, b = blockIdx.z / g.nz;
    const HeliSlice s = heli_slices<M>(tab, g)[iz];
    if (!heli_slice_ok<M>(tab, g, s, status)) return;
    const unsigned is = blockIdx.x * kHeliThreads + threadIdx.x;
    if (is >= g.ns) return;
    const unsigned iv = blockIdx.y;
    const HeliChan c = reinterpret_cast<const HeliChan*>(tab + 1)[is];
    out[b * g.out_item + (static_cast<size_t>(iz) * g.vpr + iv) * g.ns + is] =
        static_cast<T>(heli_exact<T, M>(in + b * g.in_item, g, s, c, iv, is, status + blockIdx.z));
}

// ---- FP32 fast path (T = float) ---------------------------------------------
// The only discontinuous decisions of a sample are its row range (floor/ceil
// of the projected slab edges, usability) and, for 180LI, the complementary
// ray's integer view and wrap.  The fast path
//   * evaluates the slab edges in FP32 from per-(slice, view) quotients that
//     one thread of the block forms in FP64 with the reference's operations;
//     their FP32 error stays below 1e-4 rows, so wherever an edge lies more
//     than kEdgeGuard from an integer the FP32 decision is the reference's,
//     and any other sample is recomputed by heli_exact;
//   * takes the 180LI view offset from the host split dif = dif_i + f: with
//     f in [1e-6, 1 - 1e-6] (else the channel runs heli_exact) and views below
//     2^20, the reference's rounded cur - dif lies strictly inside
//     (cur - dif_i - 1, cur - dif_i), so its floor, ceil and wraps are integer
//     arithmetic here, and its interpolation weight is 1 - f to 1e-10;
//   * sums the rows and interpolates in FP32 (the reference: FP64), which keeps
//     every output within a few FP32 ulps of the reference's.

// An FP32 slab edge x is trusted when it lies farther than
// kEdgeGuard + (|x| + |center_t|) * kEdgeGuardRel from every integer: the FP32
// error of the edges is below 2e-5 rows + 4e-7 * (|x| + |center_t|).
constexpr float kEdgeGuard = 1.0f / 16384.0f;
constexpr float kEdgeGuardRel = 1.0f / 1048576.0f;

// Per-channel FP32 section of the table (after the slices).
struct HeliChanF {
    float g;      // cos(gamma) * dsd: rows per unit of (z_dif +- thickness/2) / dso
    float h;      // cos(gamma) * dsd / dso: rows per mm of z_dif
    float difcm;  // 180LI: dif * couch_mov, the complementary ray's z offset before wrapping
    float u;      // 180LI: 1 - frac(dif), the right view's weight
    float v;      // 180LI: sc - floor(sc), the right channel's weight
    int dif_i;    // 180LI: floor(dif)
    int cl, cr;   // 180LI: floor(sc), ceil(sc); cl = -1 when the mirrored channel is off the detector
    int exact;    // 180LI: frac(dif) within 1e-6 of 0 or 1: samples of this channel run heli_exact
    int pad;
};
static_assert(sizeof(HeliChanF) == 40, "table layout");

// One (slice, view) row of the table's last section, formed once per geometry
// by heli_rows_kernel with the reference's FP64 operations.
struct HeliRowF {
    double at_d[4];          // (z_dif +- thickness/2) / dso, exact: measured view top/bottom, paired view (360LI)
    double zrel;             // z - couch_begin
    float at, ab, at2, ab2;  // the same, rounded
    float zd, wcur, wcor;    // z_dif; 360LI: the z interpolation weights
    int cur, cor;
    int pad;
};
static_assert(sizeof(HeliRowF) == 80, "table layout");

template <int M>
__device__ __forceinline__ const HeliRowF* heli_rows_f(const HeliHeader* tab, const HeliGeo& g)
{
    const HeliChanF* cf = reinterpret_cast<const HeliChanF*>(heli_slices<M>(tab, g) + g.nz);
    return reinterpret_cast<const HeliRowF*>(cf + g.ns);
}

// The per-row section: one thread per (slice, view) of a valid slice.
template <int M>
__global__ void heli_rows_kernel(HeliHeader* tab, HeliGeo g)
{
    const unsigned long long i = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<unsigned long long>(g.nz) * g.vpr) return;
    const unsigned iz = static_cast<unsigned>(i / g.vpr), iv = static_cast<unsigned>(i % g.vpr);
    const HeliSlice s = heli_slices<M>(tab, g)[iz];
    HeliRowF row{};
    if (s.valid) {
        const double zrel = __dsub_rn(s.z, g.couch_begin);
        int cur = s.first + static_cast<int>(iv);
        if (M == CTR_HELICAL_180 && cur > s.hi) cur -= static_cast<int>(g.vpr);
        const double zd = __dsub_rn(zrel, __dmul_rn(static_cast<double>(cur), g.couch_mov));
        row.cur = cur;
        row.zrel = zrel;
        row.zd = static_cast<float>(zd);
        row.at_d[0] = __ddiv_rn(__dadd_rn(zd, g.half_th), g.dso);
        row.at_d[1] = __ddiv_rn(__dsub_rn(zd, g.half_th), g.dso);
        row.at = static_cast<float>(row.at_d[0]);
        row.ab = static_cast<float>(row.at_d[1]);
        if (M == CTR_HELICAL_360) {
            const int cor = cur >= s.center ? cur - static_cast<int>(g.vpr) : cur + static_cast<int>(g.vpr);
            const double zd2 = __dsub_rn(zrel, __dmul_rn(static_cast<double>(cor), g.couch_mov));
            row.cor = cor;
            row.at_d[2] = __ddiv_rn(__dadd_rn(zd2, g.half_th), g.dso);
            row.at_d[3] = __ddiv_rn(__dsub_rn(zd2, g.half_th), g.dso);
            row.at2 = static_cast<float>(row.at_d[2]);
            row.ab2 = static_cast<float>(row.at_d[3]);
            row.wcur = static_cast<float>(-zd2 / (zd - zd2));
            row.wcor = static_cast<float>(zd / (zd - zd2));
        }
    }
    const_cast<HeliRowF*>(heli_rows_f<M>(tab, g))[i] = row;
}

__device__ __forceinline__ bool near_int(float x, float ct)
{
    return fabsf(x - rintf(x)) < kEdgeGuard + (fabsf(x) + ct) * kEdgeGuardRel;
}

// An exact FP64 edge as an FP32 value with the same floor, ceil and order
// against every integer: the integer itself, or the midpoint of its cell.
__device__ __forceinline__ float snap_edge(double x)
{
    const double f = floor(x);
    return static_cast<float>(f == x ? x : f + 0.5);
}

// The reference's edge ct - (q * cos(gamma)) * dsd for an exact quotient q.
__device__ __forceinline__ float exact_edge(const HeliGeo& g, double q, double cg)
{
    return snap_edge(__dsub_rn(g.center_t, __dmul_rn(__dmul_rn(q, cg), g.dsd)));
}

// Rows [r0, r1) from FP32 slab edges already known to be away from integers.
__device__ __forceinline__ bool rows_f(float top, float bot, float nt, int& r0, int& r1)
{
    if (bot < 0.0f || top >= nt) return false;
    r0 = static_cast<int>(floorf(fmaxf(top, 0.0f)));
    r1 = static_cast<int>(ceilf(fminf(bot, nt)));
    return true;
}

__device__ __forceinline__ float mean_f(const float* __restrict__ col, unsigned ns, int r0, int r1)
{
    float acc = 0.0f;
    for (int r = r0; r < r1; ++r) acc += __ldg(col + static_cast<size_t>(r) * ns);
    return __fdividef(acc, static_cast<float>(r1 - r0));  // within 2 ulp; 0/0 stays NaN
}

__device__ __forceinline__ float at_f(const float* __restrict__ in, const HeliGeo& g, int view, int r, int c,
                                      bool& outside)
{
    if (view < 0 || static_cast<unsigned>(view) >= g.na) {
        outside = true;
        return 0.0f;
    }
    return __ldg(in + (static_cast<size_t>(view) * g.nt + r) * g.ns + c);
}

// One output sample of the fast path, written to *o.
template <int M>
__device__ __forceinline__ void heli_fast_one(const float* __restrict__ in, float* o, const HeliHeader* tab,
                                              const HeliGeo& g, const HeliSlice& s, const HeliRowF& row,
                                              const HeliChanF& cf, unsigned iv, unsigned is, unsigned* status)
{
    const float ct = g.ct_f, nt = g.nt_f;
    const size_t view_stride = static_cast<size_t>(g.nt) * g.ns;

    if (M == CTR_HELICAL_180 && cf.exact) {  // complementary view offset too close to an integer
        const HeliChan c = reinterpret_cast<const HeliChan*>(tab + 1)[is];
        *o = static_cast<float>(heli_exact<float, M>(in, g, s, c, iv, is, status));
        return;
    }
    const float cta = fabsf(ct);
    float top = ct - row.at * cf.g, bot = ct - row.ab * cf.g;
    if (near_int(top, cta) || near_int(bot, cta)) {  // rare: the reference's edges, exactly
        const double cg = reinterpret_cast<const HeliChan*>(tab + 1)[is].cg;
        top = exact_edge(g, row.at_d[0], cg);
        bot = exact_edge(g, row.at_d[1], cg);
    }
    float top2, bot2, zd2 = 0.0f;
    int k = 0;
    if (M == CTR_HELICAL_360) {
        top2 = ct - row.at2 * cf.g;
        bot2 = ct - row.ab2 * cf.g;
        if (near_int(top2, cta) || near_int(bot2, cta)) {
            const double cg = reinterpret_cast<const HeliChan*>(tab + 1)[is].cg;
            top2 = exact_edge(g, row.at_d[2], cg);
            bot2 = exact_edge(g, row.at_d[3], cg);
        }
    } else {
        // complementary view: k - f with k = cur - dif_i, wrapped into [lo, hi] as the reference wraps cv
        k = row.cur - cf.dif_i;
        int wrap = 0;
        if (k <= s.lo) { k += static_cast<int>(g.vpr); wrap += 1; }
        if (k > s.hi) { k -= static_cast<int>(g.vpr); wrap -= 1; }
        zd2 = row.zd + cf.difcm - static_cast<float>(wrap) * g.vprcm_f;
        const float hth = g.hth_f;
        top2 = ct - (zd2 + hth) * cf.h;
        bot2 = ct - (zd2 - hth) * cf.h;
        if (near_int(top2, cta) || near_int(bot2, cta)) {
            // the reference's complementary ray: cv = cur - dif wrapped, zd2 = zrel - cv * couch_mov
            const HeliChan c = reinterpret_cast<const HeliChan*>(tab + 1)[is];
            double cv = __dsub_rn(static_cast<double>(row.cur), c.dif);
            if (cv < static_cast<double>(s.lo)) cv = __dadd_rn(cv, static_cast<double>(g.vpr));
            if (cv > static_cast<double>(s.hi)) cv = __dsub_rn(cv, static_cast<double>(g.vpr));
            const double zdd = __dsub_rn(row.zrel, __dmul_rn(cv, g.couch_mov));
            top2 = exact_edge(g, __ddiv_rn(__dadd_rn(zdd, g.half_th), g.dso), c.cg);
            bot2 = exact_edge(g, __ddiv_rn(__dsub_rn(zdd, g.half_th), g.dso), c.cg);
        }
    }
    int r0 = 0, r1 = 0;
    float vcur = 0.0f, vcor = 0.0f;
    const bool ucur = rows_f(top, bot, nt, r0, r1);
    if (ucur) vcur = mean_f(in + row.cur * view_stride + is, g.ns, r0, r1);
    const bool ucor = rows_f(top2, bot2, nt, r0, r1);
    float val;
    if (M == CTR_HELICAL_360) {
        if (ucor) vcor = mean_f(in + row.cor * view_stride + is, g.ns, r0, r1);
        val = ucur && ucor ? row.wcor * vcor + row.wcur * vcur : (ucur ? vcur : vcor);
    } else {
        if (ucor) {
            if (cf.cl < 0) {  // mirrored channel off the detector: no interpolation
                *o = vcur;
                return;
            }
            const int vl = k - 1, vr = k;
            const float w = 1.0f - cf.v;
            float left = 0.0f, right = 0.0f;
            if (vl >= 0 && static_cast<unsigned>(vr) < g.na) {
                const float* pl = in + static_cast<size_t>(vl) * view_stride + static_cast<size_t>(r0) * g.ns;
                const float* pr = pl + view_stride;
                const int dc = cf.cr - cf.cl;
                for (int r = r0; r < r1; ++r, pl += g.ns, pr += g.ns) {
                    left += w * __ldg(pl + cf.cl) + cf.v * __ldg(pl + cf.cl + dc);
                    right += w * __ldg(pr + cf.cl) + cf.v * __ldg(pr + cf.cl + dc);
                }
            } else {  // a view outside the scan (only beside a slice whose first view is 0)
                bool outside = false;
                for (int r = r0; r < r1; ++r) {
                    left += w * at_f(in, g, vl, r, cf.cl, outside) + cf.v * at_f(in, g, vl, r, cf.cr, outside);
                    right += w * at_f(in, g, vr, r, cf.cl, outside) + cf.v * at_f(in, g, vr, r, cf.cr, outside);
                }
                if (outside) atomicOr(status, CTR_HELICAL_OUTSIDE);
            }
            vcor = __fdividef((1.0f - cf.u) * left + cf.u * right, static_cast<float>(r1 - r0));
        }
        val = ucur && ucor ? __fdividef(row.zd * vcor - zd2 * vcur, row.zd - zd2) : (ucur ? vcur : vcor);
    }
    if (!ucur && !ucor) {
        atomicOr(status, CTR_HELICAL_NO_ROWS);  // the reference throws "No row data available!"
        val = 0.0f;
    }
    *o = val;
}

// Views per block of the fast kernel: a block covers kHeliThreads channels of
// kHeliViews consecutive output views of one slice.
constexpr int kHeliViews = 16;

template <int M>
__global__ void __launch_bounds__(kHeliThreads, M == CTR_HELICAL_360 ? 8 : 6)
    helical_fast_f32(const float* __restrict__ in, float* __restrict__ out, const HeliHeader* __restrict__ tab,
                     HeliGeo g, unsigned* status)
{
    const unsigned iz = blockIdx.z % g.nz, b = blockIdx.z / g.nz;
    const HeliSlice s = heli_slices<M>(tab, g)[iz];
    if (!heli_slice_ok<M>(tab, g, s, status)) return;
    const unsigned is = blockIdx.x * kHeliThreads + threadIdx.x;
    if (is >= g.ns) return;
    in += b * g.in_item;
    status += blockIdx.z;
    const HeliChanF cf = reinterpret_cast<const HeliChanF*>(heli_slices<M>(tab, g) + g.nz)[is];
    const unsigned v0 = blockIdx.y * kHeliViews, v1 = min(v0 + kHeliViews, g.vpr);
    const HeliRowF* rows = heli_rows_f<M>(tab, g) + static_cast<size_t>(iz) * g.vpr;
    float* o = out + b * g.out_item + static_cast<size_t>(iz) * g.vpr * g.ns + is;
    for (unsigned iv = v0; iv < v1; ++iv)
        heli_fast_one<M>(in, o + static_cast<size_t>(iv) * g.ns, tab, g, s, rows[iv], cf, iv, is, status);
}

// ---- 360LI, FP32: rows decided once per 32 channels ----------------------------
// Along a row of channels cos(gamma) changes slowly, so over 32 channels a slab
// edge lies in one or two cells of the detector rows.  A warp takes 32 channels
// of kH3Views views x kH3Slices slices: lane t first decides task t (one view of
// one slice) for all its channels from the extremes of cos(gamma) over them, the
// ends of an edge's range away from integers by the guard of near_int.  Then the
// warp takes the tasks one by one.  Where both edges stay in one cell a task is
// a few coalesced row loads and one multiplication a sample.  Where an edge
// passes from a cell to the next, each lane compares its edge with the one
// integer between them (lanes within the guard of it send the task to
// heli_fast_one, as do the tasks at the detector's ends).  The slices of a view
// follow one another, since the slabs of neighbouring slices share most of
// their rows (L1).  Latency and issue bound: a scan of 128 slices x 1152 views x
// 736 channels takes 340 us, 858 us sample by sample (157 -> 73 instructions a
// sample).  The samples left in a second kernel, from a list in scratch: 413 us;
// besides that, branches in place of the predicated loads 450 us, one task at a
// time in order 543 us, 8 blocks an SM (63 registers) 501 us.
constexpr int kH3Views = 4, kH3Slices = 8, kH3Warps = 4, kH3Group = 2;
static_assert(kH3Views * kH3Slices == 32, "a task a lane");

// *p where n > K (x < 0), else 0: predicated loads, where a branch would wait for
// each load before the next is issued.
template <int K>
__device__ __forceinline__ float ldg_above(const float* p, int n)
{
    float v;
    asm("{\n\t.reg .pred q;\n\tsetp.gt.s32 q, %2, %3;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}"
        : "=f"(v)
        : "l"(p), "r"(n), "n"(K));
    return v;
}
__device__ __forceinline__ float ldg_above_n(const float* p, int n, int k)
{
    float v;
    asm("{\n\t.reg .pred q;\n\tsetp.gt.s32 q, %2, %3;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}"
        : "=f"(v)
        : "l"(p), "r"(n), "r"(k));
    return v;
}
__device__ __forceinline__ float ldg_negative(const float* p, float x)
{
    float v;
    asm("{\n\t.reg .pred q;\n\tsetp.lt.f32 q, %2, 0f00000000;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}"
        : "=f"(v)
        : "l"(p), "f"(x));
    return v;
}

// One edge of a slab over the channels: the rows that all of them use start (top)
// or end (bottom) at row `all`; a lane's edge lies k - a g past the integer
// `all` (k = 1 or -1 and a = 0 where no lane's lies on its other side).
struct H3Edge {
    float k, a;
    int all;
    bool two, sure;  // the channels' edges lie on both sides of `all`; or not decided here
};

enum H3Kind { kH3None, kH3Rows, kH3Mixed, kH3Two, kH3Slow };
// One sample's rows for all channels: `at` the element of the first row that all
// of them use (channel 0), n rows; w the z weight (kH3Rows: over n); the output
// element of channel 0; the edges.
struct H3View {
    unsigned at;
    int n;
    float w;
    unsigned out;
    float tk, ta, bk, ba;
};
static_assert(sizeof(H3View) == 32, "16-byte loads");

// An edge that lies in [lo, hi] over the channels, at k - a g past a lane's integer.
__device__ __forceinline__ H3Edge h3_edge(const HeliGeo& g, float a, float lo, float hi, float guard, bool top)
{
    const float fl = floorf(lo), fh = floorf(hi);
    // all edges clamped to the detector's end: floor(max(x, 0)) = 0, ceil(min(x, nt)) = nt
    const bool clamped = top ? hi < 1.0f - guard : lo > g.nt_f - 1.0f + guard;
    H3Edge e;
    const bool away = lo - fl > guard && fh + 1.0f - hi > guard;
    const bool two = !clamped && fh == fl + 1.0f;
    e.two = two;
    e.sure = clamped || (away && (fh == fl || two));
    const float row = top ? (clamped ? 0.0f : fh) : (clamped ? g.nt_f : (two ? fh : fl + 1.0f));
    e.all = static_cast<int>(row);
    e.k = two ? g.ct_f - row : (top ? 1.0f : -1.0f);
    e.a = two ? a : 0.0f;
    return e;
}

// The rows of one sample's slab with the quotients a (top) and b (bottom), x =
// ct - a g less up to `more` over the channels' g in [g0, g1]: false where they
// are left to heli_fast_one, no rows (t.all = 0, e.all = -1) where it misses for
// all.  A lane's slab that misses where another's does not has no rows either:
// its bottom edge lies below row 0 or its top edge past the last one.
__device__ __forceinline__ bool h3_rows(const HeliGeo& g, float a, float b, float g0, float g1, float more, float guard,
                                        H3Edge& t, H3Edge& e)
{
    t = e = H3Edge{0.0f, 0.0f, 0, false, true};
    t.k = 1.0f;
    e.k = -1.0f;
    e.all = -1;
    const float t0 = g.ct_f - a * g0, t1 = g.ct_f - a * g1, b0 = g.ct_f - b * g0, b1 = g.ct_f - b * g1;
    const float up = fmaxf(more, 0.0f), down = fminf(more, 0.0f);
    const float tl = fminf(t0, t1) - up, th = fmaxf(t0, t1) - down, bl = fminf(b0, b1) - up, bh = fmaxf(b0, b1) - down;
    if (bh < -guard || tl >= g.nt_f + guard) return true;  // misses for every channel
    t = h3_edge(g, a, tl, th, guard, true);
    e = h3_edge(g, b, bl, bh, guard, false);
    return t.sure && e.sure && e.all >= t.all;
}

// A sample that its task left.  Out of line: its registers would halve the
// kernel's blocks an SM.
template <int M>
__device__ __noinline__ void h3_slow(const float* in, float* out, const HeliHeader* tab, const HeliGeo& g,
                                     unsigned* status, unsigned iz, unsigned iv, unsigned is)
{
    const HeliSlice* slices = heli_slices<M>(tab, g);
    const HeliChanF cf = reinterpret_cast<const HeliChanF*>(slices + g.nz)[is];
    const size_t row = static_cast<size_t>(iz) * g.vpr + iv;
    heli_fast_one<M>(in, out + row * g.ns + is, tab, g, slices[iz],
                                   heli_rows_f<M>(tab, g)[row], cf, iv, is, status + iz);
}

__global__ void __launch_bounds__(32 * kH3Warps, 12)
    helical_360_f32(const float* __restrict__ in, float* __restrict__ out, const HeliHeader* __restrict__ tab,
                    const __grid_constant__ HeliGeo g, unsigned* status, int slice_groups, unsigned chunks)
{
    __shared__ __align__(16) H3View s_view[2][kH3Warps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned b = blockIdx.z / slice_groups, group = blockIdx.z - b * slice_groups, iz0 = group * kH3Slices;
    const unsigned chunk = blockIdx.x * kH3Warps + warp, c0 = chunk * 32;
    if (chunk >= chunks) return;  // warp-uniform
    const unsigned is = min(c0 + lane, g.ns - 1);
    in += b * g.in_item;
    out += b * g.out_item;
    status += b * g.nz;
    if (tab->method != CTR_HELICAL_360 || tab->ns != g.ns || tab->nz != g.nz || tab->vpr != g.vpr) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && iz0 == 0) atomicOr(status, CTR_HELICAL_BAD_TABLE);
        return;
    }
    const HeliSlice* slices = heli_slices<CTR_HELICAL_360>(tab, g);
    const float gc = reinterpret_cast<const HeliChanF*>(slices + g.nz)[is].g;
    const HeliRowF* rows = heli_rows_f<CTR_HELICAL_360>(tab, g);
    float g0 = gc, g1 = gc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g0 = fminf(g0, __shfl_xor_sync(0xffffffffu, g0, o));
        g1 = fmaxf(g1, __shfl_xor_sync(0xffffffffu, g1, o));
    }
    // near_int's guard for any edge on the detector (within one row of it)
    const float guard = kEdgeGuard + (g.nt_f + 1.0f + fabsf(g.ct_f)) * kEdgeGuardRel;
    const bool on = c0 + lane < g.ns;
    const unsigned ns = g.ns;
    const unsigned iz = iz0 + lane % kH3Slices;
    bool valid = false;
    if (iz < g.nz) {
        valid = slices[iz].valid;
        if (!valid && c0 == 0 && blockIdx.y == 0)  // the reference throws before touching this slice
            atomicOr(status + iz, CTR_HELICAL_NO_VIEWS);
    }
    const unsigned iv = blockIdx.y * kH3Views + lane / kH3Slices;
    int kind = kH3None;
    if (valid && iv < g.vpr) {
        const HeliRowF& r = rows[static_cast<size_t>(iz) * g.vpr + iv];
        H3Edge t1, b1, t2, b2;
        const bool sure = h3_rows(g, r.at, r.ab, g0, g1, 0.0f, guard, t1, b1) &&
                          h3_rows(g, r.at2, r.ab2, g0, g1, 0.0f, guard, t2, b2);
        const bool hit1 = b1.all >= 0, hit2 = b2.all >= 0;
        const bool mixed = t1.two || b1.two || t2.two || b2.two;
        kind = !sure || !(hit1 || hit2) ? kH3Slow : hit1 && hit2 ? kH3Two : mixed ? kH3Mixed : kH3Rows;
        auto view = [&](int i, int from, const H3Edge& top, const H3Edge& bot, float w) {
            H3View v;
            v.n = bot.all - top.all;
            v.at = (static_cast<unsigned>(from) * g.nt + top.all) * g.ns;
            v.w = kind == kH3Rows ? __fdividef(1.0f, static_cast<float>(v.n)) : w;
            v.out = (iz * g.vpr + iv) * g.ns;
            v.tk = top.k;
            v.ta = top.a;
            v.bk = bot.k;
            v.ba = bot.a;
            s_view[i][warp][lane] = v;
        };
        if (hit1) view(0, r.cur, t1, b1, hit2 ? r.wcur : 1.0f);
        if (hit2) view(hit1 ? 1 : 0, r.cor, t2, b2, hit1 ? r.wcor : 1.0f);
    }
    unsigned m_rows = __ballot_sync(0xffffffffu, kind == kH3Rows);
    unsigned m_mixed = __ballot_sync(0xffffffffu, kind == kH3Mixed);
    unsigned m_two = __ballot_sync(0xffffffffu, kind == kH3Two);
    unsigned slow = __ballot_sync(0xffffffffu, kind == kH3Slow);
    __syncwarp();
    // the next tasks of a class, the last one again where there are fewer (the
    // repeated ones write the same value)
    auto take = [](unsigned& m, int (&k)[kH3Group]) {
#pragma unroll
        for (int u = 0; u < kH3Group; ++u) {
            k[u] = __ffs(m) - 1;
            const unsigned rest = m & (m - 1);
            if (u == kH3Group - 1 || rest) m = rest;
        }
    };
    auto sum = [&](unsigned at, int n) {
        float s = (ldg_above<0>(in + at, n) + ldg_above<1>(in + (at + ns), n)) +
                  (ldg_above<2>(in + (at + 2 * ns), n) + ldg_above<3>(in + (at + 3 * ns), n));
        for (int r = 4; r < n; ++r) s += __ldg(in + (at + r * ns));
        return s;
    };
    // the mean of a lane's rows, of which it may have none; near: a lane's edge
    // is too close to the integer
    auto mean = [&](const H3View& v, int& n, bool& near) {
        const float dt = fmaf(-v.ta, gc, v.tk), db = fmaf(v.ba, gc, -v.bk);  // minus what b lies past its integer
        near = near || fminf(fabsf(dt), fabsf(db)) < guard;
        const unsigned at = v.at + is;
        const float s = (ldg_negative(in + (at - ns), dt) + ldg_negative(in + (at + v.n * ns), db)) + sum(at, v.n);
        n = v.n + (dt < 0.0f ? 1 : 0) + (db < 0.0f ? 1 : 0);
        return __fdividef(s, static_cast<float>(n));
    };
    while (m_rows) {
        int k[kH3Group];
        take(m_rows, k);
        float v[kH3Group];
        unsigned to[kH3Group];
#pragma unroll
        for (int u = 0; u < kH3Group; ++u) {
            const uint4 t = *reinterpret_cast<const uint4*>(&s_view[0][warp][k[u]]);
            v[u] = __uint_as_float(t.z) * sum(t.x + is, static_cast<int>(t.y));
            to[u] = t.w + is;
        }
#pragma unroll
        for (int u = 0; u < kH3Group; ++u)
            if (on) out[to[u]] = v[u];
    }
    while (m_mixed) {
        int k[kH3Group];
        take(m_mixed, k);
        float v[kH3Group];
        bool near[kH3Group];
#pragma unroll
        for (int u = 0; u < kH3Group; ++u) {
            int n;
            near[u] = false;
            v[u] = mean(s_view[0][warp][k[u]], n, near[u]);
            near[u] = near[u] || n < 1;  // no row at all
        }
#pragma unroll
        for (int u = 0; u < kH3Group; ++u) {
            if (__any_sync(0xffffffffu, near[u])) slow |= 1u << k[u];
            else if (on) out[s_view[0][warp][k[u]].out + is] = v[u];
        }
    }
    for (; m_two; m_two &= m_two - 1) {
        const int k = __ffs(m_two) - 1;
        bool near = false;
        const H3View a = s_view[0][warp][k], c = s_view[1][warp][k];
        int na, nc;
        const float ma = mean(a, na, near), mc = mean(c, nc, near);
        if (__any_sync(0xffffffffu, near || na + nc < 1)) slow |= 1u << k;
        else if (on) out[a.out + is] = na < 1 ? mc : nc < 1 ? ma : fmaf(c.w, mc, a.w * ma);
    }
    for (; slow && on; slow &= slow - 1) {  // sample by sample
        const int k = __ffs(slow) - 1;
        h3_slow<CTR_HELICAL_360>(in, out, tab, g, status, iz0 + k % kH3Slices, blockIdx.y * kH3Views + k / kH3Slices, is);
    }
}

// ---- 180LI, FP32: complementary rays along their views --------------------------
// The complementary ray of output view `cur` and channel is lies dif(is) views
// back, between views k - 1 and k = cur - floor(dif), wrapped into the slice's
// views, at the mirrored channel.  dif changes by half a view from channel to
// channel, so the rays of 32 channels at one output view lie in ~14 views, and
// every load touches as many rows.  A warp takes 32 channels (one a lane) of
// kH8Views output views of a slice instead in three steps: the measured samples,
// output view by output view, into shared memory; the complementary ones, view k
// by view k (a lane's output view is k + floor(dif), idle where that is not of
// the group), where the lanes' channels are adjacent and the sum over view k's
// rows is the next step's sum over view k - 1 while the rows stay the same; then
// the interpolated rows out.  Detector rows are decided as in helical_360_f32;
// a lane's complementary edges also depend on its fraction of dif.  A view's
// rows are kept as a window of NR registers a lane, of which it sums its own.
// 128 slices x 1152 views x 736 channels: 1815 -> 1172 us, issue at 70 % of the slots:
// the complementary samples take 630 us of them, the measured ones 340 (two views
// at a time; 410 one by one, 8 at a time spill: 1305 us in all).  With each
// lane's sums formed from memory instead of a window 1523 us, a branch per row
// count 1280 us, the next window's loads a step ahead 1294 us (spills), 64 views
// a warp 1660 us, 10 blocks an SM spilled.
constexpr int kH8Views = 32, kH8Warps = 4, kH8Group = 2;
static_assert(kH8Views == 32, "a view a lane, a lane's views in a 32-bit mask");

template <int NR>
__global__ void __launch_bounds__(32 * kH8Warps, 8)
    helical_180_f32(const float* __restrict__ in, float* __restrict__ out, const HeliHeader* __restrict__ tab,
                    const __grid_constant__ HeliGeo g, unsigned* status, unsigned chunks)
{
    extern __shared__ __align__(16) float s_dyn[];  // per warp: values [view][lane], 32 tasks, z distances
    constexpr int kWarpFloats = kH8Views * 32 + 32 * 8 + kH8Views;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* s_val = s_dyn + warp * kWarpFloats;
    H3View* s_task = reinterpret_cast<H3View*>(s_val + kH8Views * 32);
    float* s_zd = s_val + kH8Views * 32 + 32 * 8;
    const unsigned b = blockIdx.z / g.nz, iz = blockIdx.z - b * g.nz;
    const unsigned chunk = blockIdx.x * kH8Warps + warp, c0 = chunk * 32;
    if (chunk >= chunks) return;  // warp-uniform
    const HeliSlice s = heli_slices<CTR_HELICAL_180>(tab, g)[iz];
    if (!heli_slice_ok<CTR_HELICAL_180>(tab, g, s, status)) return;
    in += b * g.in_item;
    out += b * g.out_item;
    status += b * g.nz;
    const bool on = c0 + lane < g.ns;
    const unsigned is = min(c0 + lane, g.ns - 1), ns = g.ns;
    const unsigned iv0 = blockIdx.y * kH8Views;
    const int nv = min(static_cast<int>(g.vpr - iv0), kH8Views), vpr = static_cast<int>(g.vpr);
    const HeliChanF cf = reinterpret_cast<const HeliChanF*>(heli_slices<CTR_HELICAL_180>(tab, g) + g.nz)[is];
    const HeliRowF* rows = heli_rows_f<CTR_HELICAL_180>(tab, g) + static_cast<size_t>(iz) * g.vpr;
    const float cm = g.vprcm_f / static_cast<float>(vpr);  // couch travel of a view
    float g0 = cf.g, g1 = cf.g, h0 = cf.h, h1 = cf.h;
    int d0 = cf.dif_i, d1 = cf.dif_i;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g0 = fminf(g0, __shfl_xor_sync(0xffffffffu, g0, o));
        g1 = fmaxf(g1, __shfl_xor_sync(0xffffffffu, g1, o));
        h0 = fminf(h0, __shfl_xor_sync(0xffffffffu, h0, o));
        h1 = fmaxf(h1, __shfl_xor_sync(0xffffffffu, h1, o));
        d0 = min(d0, __shfl_xor_sync(0xffffffffu, d0, o));
        d1 = max(d1, __shfl_xor_sync(0xffffffffu, d1, o));
    }
    const float guard = kEdgeGuard + (g.nt_f + 1.0f + fabsf(g.ct_f)) * kEdgeGuardRel;
    unsigned left = on && cf.exact ? ~0u : 0u;  // this lane's samples left to h3_slow
    unsigned has = 0;                           // its views whose measured slab meets the detector

    // a task: the edges' rows over the channels, or -1 (misses) or -2 (left) in n
    auto decide = [&](float a, float bq, float q0, float q1, float more, int view, H3View& t) {
        H3Edge te, be;
        const bool sure = h3_rows(g, a, bq, q0, q1, more, guard, te, be);
        t.n = !sure ? -2 : be.all - te.all;
        t.at = (static_cast<unsigned>(view) * g.nt + te.all) * ns;
        t.tk = te.k;
        t.ta = te.a;
        t.bk = be.k;
        t.ba = be.a;
        t.out = (te.two ? 1u : 0u) | (be.two ? 2u : 0u);  // lanes differ
    };
    // rows of a lane: whether it has the one above the common ones and the one below
    auto extra = [&](const H3View& t, float gc, float off, bool& above, bool& below) {
        const float dt = fmaf(-t.ta, gc, t.tk - off), db = fmaf(-t.ba, gc, t.bk - off);
        above = dt < 0.0f;
        below = db >= 0.0f;
        return fminf(fabsf(dt), fabsf(db)) < guard;
    };

    // 1. the measured samples, G views at a time (a view alone waits for its loads)
    {
        constexpr int G = kH8Group;
        int kind = 0;  // 1 rows that every lane uses, 2 lanes differ at an edge, 3 left
        if (lane < nv) {
            const HeliRowF& r = rows[iv0 + lane];
            H3View t;
            decide(r.at, r.ab, g0, g1, 0.0f, r.cur, t);
            kind = t.n == -2 ? 3 : t.n < 0 ? 0 : t.out ? 2 : t.n > 0 ? 1 : 0;
            t.w = t.n > 0 ? __fdividef(1.0f, static_cast<float>(t.n)) : 0.0f;
            s_task[lane] = t;
            s_zd[lane] = r.zd;
        }
        unsigned m_rows = __ballot_sync(0xffffffffu, kind == 1), m_mixed = __ballot_sync(0xffffffffu, kind == 2);
        left |= __ballot_sync(0xffffffffu, kind == 3);
        has = m_rows;
        __syncwarp();
        // the next views of a class, the last one again where there are fewer
        auto take = [](unsigned& m, int (&k)[G]) {
#pragma unroll
            for (int u = 0; u < G; ++u) {
                k[u] = __ffs(m) - 1;
                const unsigned rest = m & (m - 1);
                if (u == G - 1 || rest) m = rest;
            }
        };
        auto sum = [&](unsigned at, int n) {
            float m = (ldg_above<0>(in + at, n) + ldg_above<1>(in + (at + ns), n)) +
                      (ldg_above<2>(in + (at + 2 * ns), n) + ldg_above<3>(in + (at + 3 * ns), n));
            for (int r = 4; r < n; ++r) m += __ldg(in + (at + r * ns));
            return m;
        };
        while (m_rows) {
            int k[G];
            float m[G];
            take(m_rows, k);
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const H3View& t = s_task[k[u]];
                const float all = sum(t.at + is, t.n), q = t.w * all;
                // the quotient to its last digit (6.8e-8 from FP64 as sample by sample, 7.1e-8 without)
                const float r = fmaf(fmaf(-static_cast<float>(t.n), q, all), t.w, q);
                m[u] = fabsf(q) <= 3e38f ? r : q;
            }
#pragma unroll
            for (int u = 0; u < G; ++u) s_val[k[u] * 32 + lane] = m[u];
        }
        while (m_mixed) {
            int k[G];
            float m[G];
            take(m_mixed, k);
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const H3View t = s_task[k[u]];
                const unsigned at = t.at + is;
                bool above, below;
                if (extra(t, cf.g, 0.0f, above, below)) left |= 1u << k[u];
                const int n = t.n + above + below;
                m[u] = sum(at, t.n) +
                       (ldg_above<0>(in + (at - ns), above) + ldg_above<0>(in + (at + t.n * ns), below));
                m[u] = __fdividef(m[u], static_cast<float>(n));
                has |= n > 0 ? 1u << k[u] : 0u;
            }
#pragma unroll
            for (int u = 0; u < G; ++u) s_val[k[u] * 32 + lane] = m[u];
        }
        __syncwarp();
    }

    // 2. the complementary samples: K runs over the unwrapped views cur - floor(dif)
    const int base = s.first + static_cast<int>(iv0);
    const float f = 1.0f - cf.u, off = f * cm * cf.h;  // the fraction of dif, and its way along the rows
    const unsigned cl = max(cf.cl, 0), cr = max(cf.cr, 0);
    const float w = 1.0f - cf.v;
    const int k0 = base - d1, k1 = base + nv - 1 - d0;
    const unsigned view = g.nt * ns;
    float right[NR], leftv[NR];  // the window's rows of views k and k - 1 at the lane's mirrored channel
    unsigned held = 0;  // the element that `right` starts at, and its rows
    int held_n = 0;
    for (int kb = k0; kb <= k1; kb += 32) {
        if (kb + lane <= k1) {
            int k = kb + lane;
            k += k < s.lo ? vpr : (k > s.hi ? -vpr : 0);
            const int ivk = k - s.first + (k < s.first ? vpr : 0);
            const float zd = rows[ivk].zd;
            H3View t;
            decide(zd + g.hth_f, zd - g.hth_f, h0, h1, cm * h1, k, t);
            // the window: the common rows and, where lanes differ at an edge (k away from 1 and -1), the one beyond
            const unsigned above = t.out & 1u, below = t.out >> 1;
            if (t.n >= 0) {
                t.at -= above * ns;
                t.n += above + below;
                if (t.n > NR) t.n = -2;
            }
            if (k == 0) t.n = -2;  // view k - 1 lies before the scan
            t.w = zd;
            s_task[lane] = t;
        }
        __syncwarp();
        for (int j = 0; j < min(32, k1 - kb + 1); ++j) {
            const H3View t = s_task[j];
            const int v = kb + j + cf.dif_i - base;
            const bool act = static_cast<unsigned>(v) < static_cast<unsigned>(nv);
            const unsigned bit = act ? 1u << v : 0u;
            if (t.n < 1) {
                held_n = 0;
                // no complementary row: the measured sample as it is, where there is one
                left |= t.n == -2 ? bit : bit & ~has;
                continue;
            }
            auto window = [&](float (&c)[NR], unsigned at) {
                const float* p = in + (at + cl);
                const float* q = in + (at + cr);
#pragma unroll
                for (int r = 0; r < NR; ++r)  // 0 past the window
                    c[r] = fmaf(w, ldg_above_n(p + r * ns, t.n, r), cf.v * ldg_above_n(q + r * ns, t.n, r));
            };
            // (a longer one only where the lane's rows are taken one by one)
            if ((t.out ? held_n >= t.n : held_n == t.n) && held == t.at - view) {
#pragma unroll
                for (int r = 0; r < NR; ++r) leftv[r] = right[r];
            } else {
                window(leftv, t.at - view);
            }
            window(right, t.at);
            held = t.at;
            held_n = t.n;
            int n = t.n;
            float sl = leftv[0], sr = right[0];
            if (t.out) {  // the lane's rows of the window
                const float dt = fmaf(-t.ta, cf.h, t.tk - off), db = fmaf(-t.ba, cf.h, t.bk - off);
                if (fminf(fabsf(dt), fabsf(db)) < guard) left |= bit;
                const int from = (t.out & 1u) && dt >= 0.0f ? 1 : 0, to = t.n - ((t.out & 2u) && db < 0.0f ? 1 : 0);
                n = to - from;
                if (from > 0 || n < 1) sl = sr = 0.0f;
#pragma unroll
                for (int r = 1; r < NR; ++r)
                    if (r < to) {
                        sl += leftv[r];
                        sr += right[r];
                    }
            } else {
#pragma unroll
                for (int r = 1; r < NR; ++r) {
                    sl += leftv[r];
                    sr += right[r];
                }
            }
            if (n < 1) left |= bit & ~has;
            if (!act || n < 1) continue;
            const float vcor = __fdividef(fmaf(f, sl, cf.u * sr), static_cast<float>(n));
            const float zd = s_zd[v], zd2 = t.w + f * cm;
            float val = vcor;
            if (cf.cl < 0) {  // mirrored channel off the detector: no interpolation
                val = has & bit ? s_val[v * 32 + lane] : 0.0f;
            } else if (has & bit) {
                val = __fdividef(zd * vcor - zd2 * s_val[v * 32 + lane], zd - zd2);
            }
            s_val[v * 32 + lane] = val;
        }
        __syncwarp();
    }

    // 3. out
    const unsigned to = (iz * g.vpr + iv0) * ns + is;
    for (int v = 0; v < nv; ++v)
        if (on && !(left >> v & 1)) out[to + v * ns] = s_val[v * 32 + lane];
    // each lane its own next sample: the lanes' views differ
    for (left = on ? left & (~0u >> (32 - nv)) : 0u; left; left &= left - 1)
        h3_slow<CTR_HELICAL_180>(in, out, tab, g, status, iz, iv0 + __ffs(left) - 1, is);
}

size_t table_bytes(const ctr_helical_param* p)
{
    return sizeof(HeliHeader) + sizeof(HeliChan) * p->ns + sizeof(HeliSlice) * p->nz + sizeof(HeliChanF) * p->ns +
           sizeof(HeliRowF) * static_cast<size_t>(p->nz) * p->view_per_rot;
}

int check_param(const ctr_helical_param* p)
{
    if (!p) return fail(CTR_ERR_INVALID_ARG, "null helical parameters");
    if (p->ns < 1 || p->nt < 1 || p->na < 1 || p->view_per_rot < 1 || p->nz < 1)
        return fail(CTR_ERR_INVALID_ARG, "empty helical geometry");
    const double f[] = {p->ds, p->offset_s, p->offset_t, p->orbit, p->couch_begin, p->couch_mov,
                        p->dz, p->z0, p->thickness, p->dso, p->dsd};
    for (double v : f)
        if (!std::isfinite(v)) return fail(CTR_ERR_INVALID_ARG, "non-finite helical parameter");
    if (p->couch_mov == 0.0 || p->orbit == 0.0 || p->dso == 0.0 || p->dsd == 0.0 || p->ds == 0.0)
        return fail(CTR_ERR_INVALID_ARG, "couch_mov, orbit, ds, dso and dsd must be non-zero");
    if (p->view_per_rot > 65535u) return fail(CTR_ERR_UNSUPPORTED, "view_per_rot > 65535");
    return CTR_OK;
}

HeliGeo make_geo(const ctr_helical_param* p)
{
    HeliGeo g;
    g.ns = p->ns;
    g.nt = p->nt;
    g.na = p->na;
    g.vpr = p->view_per_rot;
    g.nz = p->nz;
    g.center_t = static_cast<double>(p->nt - 1) / 2.0 + p->offset_t;
    g.couch_begin = p->couch_begin;
    g.couch_mov = p->couch_mov;
    g.half_th = p->thickness / 2.0;
    g.dso = p->dso;
    g.dsd = p->dsd;
    g.nt_d = static_cast<double>(p->nt);
    g.ns_last = static_cast<double>(p->ns - 1);
    g.in_item = static_cast<size_t>(p->na) * p->nt * p->ns;
    g.out_item = static_cast<size_t>(p->nz) * p->view_per_rot * p->ns;
    g.ct_f = static_cast<float>(g.center_t);
    g.nt_f = static_cast<float>(p->nt);
    g.hth_f = static_cast<float>(g.half_th);
    g.vprcm_f = static_cast<float>(p->view_per_rot * p->couch_mov);
    return g;
}

// Conditions of the FP32 fast path: a slab whose top edge lies above its
// bottom edge on every channel (thickness >= 0, dso and dsd > 0, |gamma| below
// pi/2), views and rows far inside the ranges its integer and FP32 arithmetic
// cover.  Elsewhere T=float runs the exact kernel.
bool fast_ok(const ctr_helical_param* p)
{
    const double center_s = static_cast<double>(p->ns - 1) / 2.0 + p->offset_s;
    const double gmax = std::fmax(std::fabs((0.0 - center_s) * p->ds / p->dsd),
                                  std::fabs((static_cast<double>(p->ns - 1) - center_s) * p->ds / p->dsd));
    return p->thickness >= 0.0 && p->dso > 0.0 && p->dsd > 0.0 && gmax < kHeliPi / 2 - 1e-3 &&
           p->na < (1u << 20) && p->nt < (1u << 15) && std::fabs(p->view_per_rot * p->couch_mov) < 1e4;
}

// 360LI by tasks: false (nothing launched) where an item's elements need more
// than 32 bits.
bool launch_360(const ctr_helical_param* p, const HeliGeo& g, const float* in, float* out, const HeliHeader* tab,
                unsigned* status, int batch, cudaStream_t stream)
{
    const unsigned chunks = div_up(p->ns, 32), views = div_up(p->view_per_rot, kH3Views),
                   groups = div_up(p->nz, kH3Slices);
    if (g.in_item > 0xffffffffu || g.out_item > 0xffffffffu) return false;
    helical_360_f32<<<dim3(div_up(chunks, kH3Warps), views, groups * batch), 32 * kH3Warps, 0, stream>>>(
        in, out, tab, g, status, groups, chunks);
    return true;
}

// 180LI view by view: false (nothing launched) where an item's elements need
// more than 32 bits, a complementary ray lies a rotation or more away, or the
// slab covers more rows than the window, and for small scans.
bool launch_180(const ctr_helical_param* p, const HeliGeo& g, const float* in, float* out, const HeliHeader* tab,
                unsigned* status, int batch, cudaStream_t stream)
{
    const double center_s = static_cast<double>(p->ns - 1) / 2.0 + p->offset_s;
    for (double c : {0.0, static_cast<double>(p->ns - 1)}) {
        const double dif = (kHeliPi - 2 * (c - center_s) * p->ds / p->dsd) / p->orbit;
        if (!(dif >= 0.0 && dif <= static_cast<double>(p->view_per_rot) - 1.0)) return false;
    }
    if (g.in_item > 0xffffffffu || g.out_item > 0xffffffffu) return false;
    const unsigned chunks = div_up(p->ns, 32);
    constexpr size_t smem = sizeof(float) * kH8Warps * (kH8Views * 32 + 32 * 8 + kH8Views);
    const unsigned views = div_up(p->view_per_rot, kH8Views);
    const dim3 grid(div_up(chunks, kH8Warps), views, p->nz * batch);
    // Few warps leave the steps' latency bare: 960 warps (8 slices x 360 views x
    // 300 channels) 39 us against 31 sample by sample, 3840 warps (16 x 500 x
    // 450) 58 against 83.  An item's count, so that an item's values are the same
    // in any batch.
    if (static_cast<size_t>(chunks) * views * p->nz < 2048) return false;
    const double slab = p->thickness * p->dsd / p->dso;  // in rows, at the centre channel
    if (slab <= 2.5)
        helical_180_f32<4><<<grid, 32 * kH8Warps, smem, stream>>>(in, out, tab, g, status, chunks);
    else if (slab <= 6.0)
        helical_180_f32<8><<<grid, 32 * kH8Warps, smem, stream>>>(in, out, tab, g, status, chunks);
    else
        return false;
    return true;
}

template <typename T>
int helical_run(int method, const ctr_helical_param* p, const T* in, T* out, const void* table, unsigned* status,
                int batch, cudaStream_t stream)
{
    int st = check_param(p);
    if (st) return st;
    if (bad_ptr(in) || bad_ptr(out) || bad_ptr(table) || bad_ptr(status))
        return fail(CTR_ERR_INVALID_ARG, "null pointer");
    if ((st = check_common(batch))) return st;
    if (static_cast<unsigned long long>(p->nz) * batch > 65535ull)
        return fail(CTR_ERR_UNSUPPORTED, "nz * batch > 65535");
    const HeliGeo g = make_geo(p);
    const dim3 grid(div_up(p->ns, kHeliThreads), p->view_per_rot, p->nz * batch);
    const HeliHeader* tab = static_cast<const HeliHeader*>(table);
    if (std::is_same<T, float>::value && fast_ok(p)) {
        const float* fin = reinterpret_cast<const float*>(in);
        float* fout = reinterpret_cast<float*>(out);
        const dim3 grid(div_up(p->ns, kHeliThreads), div_up(p->view_per_rot, kHeliViews), p->nz * batch);
        const bool done = method == CTR_HELICAL_360 ? launch_360(p, g, fin, fout, tab, status, batch, stream)
                                                    : launch_180(p, g, fin, fout, tab, status, batch, stream);
        if (!done && method == CTR_HELICAL_360)
            helical_fast_f32<CTR_HELICAL_360><<<grid, kHeliThreads, 0, stream>>>(fin, fout, tab, g, status);
        else if (!done)
            helical_fast_f32<CTR_HELICAL_180><<<grid, kHeliThreads, 0, stream>>>(fin, fout, tab, g, status);
        return check_launch(method == CTR_HELICAL_360 ? "helical 360LI (FP32)" : "helical 180LI (FP32)");
    }
    if (method == CTR_HELICAL_360)
        helical_kernel<T, CTR_HELICAL_360><<<grid, kHeliThreads, 0, stream>>>(in, out, tab, g, status);
    else
        helical_kernel<T, CTR_HELICAL_180><<<grid, kHeliThreads, 0, stream>>>(in, out, tab, g, status);
    return check_launch(method == CTR_HELICAL_360 ? "helical 360LI" : "helical 180LI");
}

}  // namespace
}  // namespace ctr

using namespace ctr;

extern "C" {

size_t ctr_helical_interpolation_table_bytes(const ctr_helical_param* p)
{
    return p ? table_bytes(p) : 0;
}

int ctr_helical_interpolation_prep(const ctr_helical_param* p, int method, void* table, cudaStream_t stream)
{
    int st = check_param(p);
    if (st) return st;
    if (method != CTR_HELICAL_360 && method != CTR_HELICAL_180)
        return fail(CTR_ERR_INVALID_ARG, "helical method must be CTR_HELICAL_360 or CTR_HELICAL_180");
    if (bad_ptr(table)) return fail(CTR_ERR_INVALID_ARG, "null table");
    const size_t row_bytes = sizeof(HeliRowF) * static_cast<size_t>(p->nz) * p->view_per_rot;
    std::vector<unsigned char> host(table_bytes(p) - row_bytes);  // the rows are formed on the device
    HeliHeader* hdr = reinterpret_cast<HeliHeader*>(host.data());
    HeliChan* ch = reinterpret_cast<HeliChan*>(hdr + 1);
    HeliSlice* sl = reinterpret_cast<HeliSlice*>(ch + p->ns);
    *hdr = HeliHeader{method, p->ns, p->nz, p->view_per_rot};
    // per channel (src/helical_interpolation.cc:174-175, 196, 214)
    const double center_s = static_cast<double>(p->ns - 1) / 2.0 + p->offset_s;
    for (unsigned is = 0; is < p->ns; ++is) {
        const double s = (static_cast<double>(is) - center_s) * p->ds;
        const double gamma = s / p->dsd;
        ch[is].cg = std::cos(gamma);
        ch[is].dif = (kHeliPi - 2 * gamma) / p->orbit;
        ch[is].sc = center_s - s / p->ds;
        ch[is].pad = 0.0;
    }
    // per slice: the view range checks of src/helical_interpolation.cc:84-90 (360LI) and 160-166
    // (180LI); a failing slice is marked and reported by the kernel in its status word
    const int vpr = static_cast<int>(p->view_per_rot);
    double z = p->z0;
    for (unsigned iz = 0; iz < p->nz; ++iz, z += p->dz) {
        const double cv = std::round((z - p->couch_begin) / p->couch_mov);
        HeliSlice& s = sl[iz];
        s = HeliSlice{z, 0, 0, 0, 0, 0, 0};
        if (!(std::fabs(cv) < 1e9)) continue;  // far outside any scan: invalid
        s.center = static_cast<int>(cv);
        if (method == CTR_HELICAL_360) {
            s.lo = s.center - vpr;
            s.hi = s.center + vpr - 1;
        } else {
            s.lo = s.center - vpr / 2;
            s.hi = s.lo + vpr - 1;
        }
        if (s.lo < 0 || static_cast<unsigned>(s.hi) >= p->na) continue;
        s.valid = 1;
        s.first = method == CTR_HELICAL_360
                      ? (s.lo / vpr + 1) * vpr
                      : static_cast<int>(std::ceil(s.lo / static_cast<double>(p->view_per_rot)) * p->view_per_rot);
    }
    // the FP32 fast path's per-channel section (from the same FP64 values)
    HeliChanF* cf = reinterpret_cast<HeliChanF*>(sl + p->nz);
    for (unsigned is = 0; is < p->ns; ++is) {
        const HeliChan& c = ch[is];
        HeliChanF& f = cf[is];
        f = HeliChanF{};
        f.g = static_cast<float>(c.cg * p->dsd);
        f.h = static_cast<float>(c.cg * p->dsd / p->dso);
        f.difcm = static_cast<float>(c.dif * p->couch_mov);
        const bool finite = std::fabs(c.dif) < static_cast<double>(1 << 20);
        const double di = finite ? std::floor(c.dif) : 0.0, fr = c.dif - di;
        f.dif_i = static_cast<int>(di);
        f.u = static_cast<float>(1.0 - fr);
        f.exact = (!finite || fr < 1e-6 || fr > 1.0 - 1e-6) ? 1 : 0;
        if (c.sc < 0.0 || c.sc > static_cast<double>(p->ns - 1)) {
            f.cl = f.cr = -1;
        } else {
            f.cl = static_cast<int>(std::floor(c.sc));
            f.cr = static_cast<int>(std::ceil(c.sc));
            f.v = static_cast<float>(c.sc - f.cl);
        }
    }
    cudaError_t e = cudaMemcpyAsync(table, host.data(), host.size(), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) {
        const HeliGeo g = make_geo(p);
        const unsigned long long rows = static_cast<unsigned long long>(p->nz) * p->view_per_rot;
        if (rows > 65535ull * 65535ull) return fail(CTR_ERR_UNSUPPORTED, "nz * view_per_rot too large");
        HeliHeader* tab = static_cast<HeliHeader*>(table);
        if (method == CTR_HELICAL_360)
            heli_rows_kernel<CTR_HELICAL_360><<<div_up(rows, 256), 256, 0, stream>>>(tab, g);
        else
            heli_rows_kernel<CTR_HELICAL_180><<<div_up(rows, 256), 256, 0, stream>>>(tab, g);
        e = cudaGetLastError();
    }
    // the host vector dies on return: wait for the staged copy to leave it
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e == cudaSuccess ? CTR_OK : fail(CTR_ERR_CUDA, "helical table: %s", cudaGetErrorString(e));
}

int ctr_helical_interpolation_360_f32(const ctr_helical_param* p, const float* in, float* out, const void* table,
                                      unsigned int* status, int batch, cudaStream_t stream)
{
    return helical_run<float>(CTR_HELICAL_360, p, in, out, table, status, batch, stream);
}
int ctr_helical_interpolation_360_f64(const ctr_helical_param* p, const double* in, double* out,
                                      const void* table, unsigned int* status, int batch, cudaStream_t stream)
{
    return helical_run<double>(CTR_HELICAL_360, p, in, out, table, status, batch, stream);
}
int ctr_helical_interpolation_180_f32(const ctr_helical_param* p, const float* in, float* out, const void* table,
                                      unsigned int* status, int batch, cudaStream_t stream)
{
    return helical_run<float>(CTR_HELICAL_180, p, in, out, table, status, batch, stream);
}
int ctr_helical_interpolation_180_f64(const ctr_helical_param* p, const double* in, double* out,
                                      const void* table, unsigned int* status, int batch, cudaStream_t stream)
{
    return helical_run<double>(CTR_HELICAL_180, p, in, out, table, status, batch, stream);
}

}  // extern "C"
