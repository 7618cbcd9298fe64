// mixed.cu -- mixed-precision solve: FP32 2x2-block PCR + FP64 iterative
// refinement, and the fused FP64 pentadiagonal residual.
//
// Why blocks.  The reference's scalar PCR-Penta eliminates with off-diagonal
// pivots (alpha = -a[i]/b[i-2d], kernel.cu:73), which amplifies rounding by
// 1/|pivot|: in FP32 it loses 3-4 digits on diagonally dominant inputs, and
// an exactly zero off-diagonal breaks it outright.  Grouping rows in pairs
// turns the pentadiagonal matrix into a block-tridiagonal one with 2x2
// blocks; block PCR then pivots on the 2x2 diagonal blocks, which stay
// well conditioned for dominant systems (block cyclic reduction preserves
// block dominance and squares the coupling every stride), so the FP32 solve
// keeps ~7 digits and one refinement sweep usually reaches 1e-13.
//
// Block row k holds rows 2k, 2k+1 and reads L_k X_{k-d} + X_k + U_k X_{k+d}
// = Y_k after normalisation by its diagonal block (D = I).  One stride:
//     D' = I - L_k U_{k-d} - U_k L_{k+d},  L' = -L_k L_{k-d},
//     U' = -U_k U_{k+d},  Y' = Y_k - L_k Y_{k-d} - U_k Y_{k+d},
// then L, U, Y <- D'^{-1} (L', U', Y').  Strides stop early once every
// |L|,|U| entry of a system is below kTrunc (the couplings then change X by
// less than kTrunc*|X|, far below FP32 resolution) -- truncated PCR.
//
// FP64 budget.  GB300 issues FP64 at ~1/64 of the FP32 rate, so FP64 is kept
// to the residual (5 DFMA per row) and the correction (1 DADD per row).  Row
// scaling by the main diagonal is done by powers of two in the integer
// pipe, and every FP64<->FP32 conversion here is integer bit arithmetic
// (no F2F instructions, which also issue on the FP64 pipe).
//
// Stopping rule.  With dx_s the correction of sweep s, a system is done when
// |dx_s| <= tol/2 |x| (the correction bounds what it leaves), or when the
// corrections contract (rho = |dx_s|/|dx_{s-1}| < 0.5) and twice the
// geometric tail rho/(1-rho)|dx_s| is <= tol |x|.
// Each kernel reads the per-system norms left by the previous kernel, so the
// decision needs no host round trip; finished systems skip all later work.
#include <algorithm>
#include <cfloat>
#include <cstring>

#include "pcrp_internal.h"
#include "mixed_internal.h"
#include "mixed_dev.cuh"
#include "tma.cuh"

namespace pcrp {
namespace {

constexpr int kMpThreads = 256;
constexpr int kMpTryThreads = 256;
static_assert(kMpTile % kMpThreads == 0 && kMpThreads % 2 == 0, "refinement tiles: whole rows per thread, pairs in adjacent lanes");

// Row i of system j of an iterate: at j*ss + i*rs, or (ragged output, rg
// non-null) at rg[j].x + i for i < rg[j].y; padding rows read as zero and
// are not stored.
__device__ __forceinline__ double x_read(const double* __restrict__ x, int64_t ss, int64_t rs,
                                         const longlong2* __restrict__ rg, int64_t j, int64_t i)
{
    if (!rg) return x[j * ss + i * rs];
    const longlong2 g = __ldg(rg + j);
    return i < g.y ? x[g.x + i] : 0.0;
}

__device__ __forceinline__ void x_write(double* __restrict__ x, int64_t ss, int64_t rs,
                                        const longlong2* __restrict__ rg, int64_t j, int64_t i, double v)
{
    if (!rg) { x[j * ss + i * rs] = v; return; }
    const longlong2 g = __ldg(rg + j);
    if (i < g.y) x[g.x + i] = v;
}

// Where sweep s reads x_{s-1} and writes x_s.  x_0 is a float (the first
// correction itself), kept as one in X0f (m*n, contiguous) when more sweeps
// follow: srcf (sweep 1) and dstf (sweep 0) then stand in for src and dst.
struct XView {
    const double* src; int64_t sss, srs; const longlong2* srg;
    double* dst; int64_t dss, drs; const longlong2* drg;
    const float* srcf; float* dstf;
};

// x_s of row i of system j (FP32 correction d), with the maxima of |dx| and
// |x| folded into dmax and xbits.
__device__ __forceinline__ void x_update(const XView& v, int64_t n, int64_t j, int64_t i, float d, float& dmax,
                                         unsigned long long& xbits)
{
    const double dd = f2d(d);
    double x = dd;
    if (v.srcf) x = __dadd_rn(f2d(v.srcf[j * n + i]), dd);
    else if (v.src) x = __dadd_rn(x_read(v.src, v.sss, v.srs, v.srg, j, i), dd);
    if (v.dstf) v.dstf[j * n + i] = d;
    else x_write(v.dst, v.dss, v.drs, v.drg, j, i, x);
    dmax = fmaxf(dmax, fabsf(d));
    xbits = max(xbits, absbits(x));
}

// Iterates of sweep s: x_0 in X0f when more sweeps follow, every later x_s in
// the output; x_{s-1} is read from where sweep s-1 wrote it.
// The output of a ragged batch is addressed through rg.
__device__ __forceinline__ XView x_view(int s, int max_sweeps, float* X0f, double* xout, int64_t oss, int64_t ors,
                                        const longlong2* rg)
{
    XView v{nullptr, oss, ors, rg, xout, oss, ors, rg, nullptr, nullptr};
    if (s == 1) v.srcf = X0f;
    else if (s > 1) v.src = xout;
    if (s == 0 && max_sweeps >= 2) v.dstf = X0f;
    return v;
}

// Graph-driven sweeps: the per-sweep fields from the device sweep counter
// (written by the previous sweep's last kernel, complete before this one
// starts).  No-ops for host-driven launches.
__device__ __forceinline__ void mp_resolve(MpArgs& p)
{
    if (p.ctr) p.sweep = *p.ctr;
}

__device__ __forceinline__ void mp_resolve(MpPassArgs& p)
{
    if (!p.ctr) return;
    const int s = *p.ctr;
    p.sweep = s;
    p.live = p.live0 + s;
    if (p.level0) p.srcY = (s & 1) ? p.R1 : p.R0;
    if (p.pre0) {
        unsigned* pre = p.pre0 + (size_t)s * kMpMaxPasses * p.m;
        p.ndx_pre_in = p.pass > 0 ? pre + (size_t)(p.pass - 1) * p.m : nullptr;
        p.ndx_pre_out = p.final_step ? nullptr : pre + (size_t)p.pass * p.m;
    }
    if (p.nx0) p.nx = p.nx0 + (size_t)s * p.m;
}

// The six FP64 values of rows i0 = 2k and i1 = 2k+1 of system j (i1 may be
// the dummy row n of an odd system).  Contiguous pairs at an even element
// offset are read as one 16-byte load per array.  A null outer band (a or e)
// is zero and not read.  In a ragged batch the rows past the system's own
// are identity rows, and the band slots of its last rows that would couple
// to them read as zero (the caller's values there are not part of the
// system).
struct PairRow { double a0, a1, b0, b1, c0, c1, d0, d1, e0, e1, y0, y1; };

// L2 residency of the band loads of sweep 0: the prep loads a tile's bands
// to keep (the residual of the same tile reads them again once its cyclic
// reduction is done), the residual loads them for the last time.
enum class Keep { normal, last, first };

__device__ __forceinline__ double2 ldg2_policy(const double* q, uint64_t pol)
{
    double2 v;
    asm("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(q), "l"(pol));
    return v;
}

__device__ __forceinline__ double2 ldg2(const double* q, Keep keep, uint64_t pol)
{
    return keep == Keep::normal ? *reinterpret_cast<const double2*>(q) : ldg2_policy(q, pol);
}

// RG: the batch is ragged (p.rg non-null); the uniform kernels are compiled
// without the ragged addressing.
template <bool RG>
__device__ __forceinline__ PairRow load_pair(const MpArgs& p, int64_t j, int64_t i0, Keep keep, bool has_a, bool has_e)
{
    PairRow P;
    int64_t n = p.n, rs = p.rs, base = j * p.ss;
    if (RG) {
        const longlong2 g = __ldg(p.rg + j);
        base = g.x; n = g.y; rs = 1;
        if (i0 >= n) {
            P = {0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            return P;
        }
    }
    const int64_t g0 = base + i0 * rs;
    const double2 z = make_double2(0.0, 0.0);
    if (p.vec && rs == 1 && ((g0 & 1) == 0) && i0 + 1 < n) {
        const uint64_t pol = keep == Keep::last ? tma::policy_evict_last()
                             : keep == Keep::first ? tma::policy_evict_first() : 0;
        const double2 a = has_a ? ldg2(p.a + g0, keep, pol) : z;
        const double2 b = ldg2(p.b + g0, keep, pol);
        const double2 c = ldg2(p.c + g0, keep, pol);
        const double2 d = ldg2(p.d + g0, keep, pol);
        const double2 e = has_e ? ldg2(p.e + g0, keep, pol) : z;
        const double2 y = ldg2(p.y + g0, keep, pol);
        P = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, e.x, e.y, y.x, y.y};
    } else {
        P.a0 = has_a ? p.a[g0] : 0.0; P.b0 = p.b[g0]; P.c0 = p.c[g0]; P.d0 = p.d[g0];
        P.e0 = has_e ? p.e[g0] : 0.0; P.y0 = p.y[g0];
        if (i0 + 1 < n) {
            const int64_t g1 = g0 + rs;
            P.a1 = has_a ? p.a[g1] : 0.0; P.b1 = p.b[g1]; P.c1 = p.c[g1]; P.d1 = p.d[g1];
            P.e1 = has_e ? p.e[g1] : 0.0; P.y1 = p.y[g1];
        } else {
            P.a1 = 0.0; P.b1 = 0.0; P.c1 = 1.0; P.d1 = 0.0; P.e1 = 0.0; P.y1 = 0.0;
        }
    }
    if (RG) {
        if (i0 + 1 >= n) P.d0 = 0.0;
        if (i0 + 2 >= n) { P.e0 = 0.0; P.d1 = 0.0; }
        if (i0 + 3 >= n) P.e1 = 0.0;
    }
    return P;
}

template <bool RG>
__device__ __forceinline__ PairRow load_pair(const MpArgs& p, int64_t j, int64_t i0, Keep keep = Keep::normal)
{
    return load_pair<RG>(p, j, i0, keep, p.a != nullptr, p.e != nullptr);
}

// The FP32 row-scaled diagonal block and couplings of block row k (rows
// i0 = 2k, i1 = 2k+1) of a system with n rows.  Row i1 = n (odd n) is a
// dummy identity row.  Out-of-range band slots are never read as values.
struct BlockRow { M2 D, L, U; float y0, y1; };

__device__ __forceinline__ BlockRow block_of(const PairRow& P, int64_t i0, int64_t n)
{
    BlockRow B;
    const int64_t i1 = i0 + 1;
    const int sh0 = d_exponent(P.c0);
    const float a0 = i0 >= 2 ? d2f_scaled(P.a0, sh0) : 0.0f;
    const float b0 = i0 >= 1 ? d2f_scaled(P.b0, sh0) : 0.0f;
    const float d0 = i0 + 1 < n ? d2f_scaled(P.d0, sh0) : 0.0f;
    const float e0 = i0 + 2 < n ? d2f_scaled(P.e0, sh0) : 0.0f;
    const float cf0 = d2f_scaled(P.c0, sh0);
    float a1 = 0.0f, b1 = 0.0f, cf1 = 1.0f, d1 = 0.0f, e1 = 0.0f;
    B.y0 = d2f_scaled(P.y0, sh0);
    B.y1 = 0.0f;
    if (i1 < n) {
        const int sh1 = d_exponent(P.c1);
        a1 = i1 >= 2 ? d2f_scaled(P.a1, sh1) : 0.0f;
        b1 = d2f_scaled(P.b1, sh1);
        cf1 = d2f_scaled(P.c1, sh1);
        d1 = i1 + 1 < n ? d2f_scaled(P.d1, sh1) : 0.0f;
        e1 = i1 + 2 < n ? d2f_scaled(P.e1, sh1) : 0.0f;
        B.y1 = d2f_scaled(P.y1, sh1);
    }
    B.D = {cf0, d0, b1, cf1};
    B.L = {a0, b0, 0.0f, a1};
    B.U = {e0, 0.0f, d1, e1};
    return B;
}

// The same for a block row with all its band slots inside the system; values
// beyond the row conversion's range take the general form.
__device__ __forceinline__ BlockRow block_inner(const PairRow& P, int64_t i0, int64_t n)
{
    const RowScale s0 = row_scale(P.c0), s1 = row_scale(P.c1);
    int top = 0;
    BlockRow B;
    B.D = {d2f_row(P.c0, s0, top), d2f_row(P.d0, s0, top), d2f_row(P.b1, s1, top), d2f_row(P.c1, s1, top)};
    B.L = {d2f_row(P.a0, s0, top), d2f_row(P.b0, s0, top), 0.0f, d2f_row(P.a1, s1, top)};
    B.U = {d2f_row(P.e0, s0, top), 0.0f, d2f_row(P.d1, s1, top), d2f_row(P.e1, s1, top)};
    B.y0 = d2f_row(P.y0, s0, top);
    B.y1 = d2f_row(P.y1, s1, top);
    if (!(s0.ok && s1.ok && row_fits(top))) B = block_of(P, i0, n);
    return B;
}

// ---------------------------------------------------------------------------
// prep: level-0 normalised block state and the first right-hand side
// ---------------------------------------------------------------------------
// One block row of the prep work: row scaling, FP32 blocks, diagonal inverse,
// the normalised couplings and rhs.
struct PrepRow { M2 L, U, Mi; float2 Y; double2 y; };   // y: the two FP64 rhs values (0 past the system)

__device__ __forceinline__ PrepRow prep_of(const BlockRow& B)
{
    PrepRow r;
    r.Mi = minv(B.D);
    r.L = mmul(r.Mi, B.L);
    r.U = mmul(r.Mi, B.U);
    r.Y = make_float2(fmaf(r.Mi.m0, B.y0, r.Mi.m1 * B.y1), fmaf(r.Mi.m2, B.y0, r.Mi.m3 * B.y1));
    return r;
}

// The inverse of the row-scaled FP32 diagonal block of a block row, as prep_of
// forms it.
__device__ __forceinline__ M2 diag_inverse(const PairRow& P, int64_t i0, int64_t n)
{
    const RowScale s0 = row_scale(P.c0), s1 = row_scale(P.c1);
    int top = 0;
    M2 D = {d2f_row(P.c0, s0, top), d2f_row(P.d0, s0, top), d2f_row(P.b1, s1, top), d2f_row(P.c1, s1, top)};
    if (i0 + 1 >= n) D = {d2f_scaled(P.c0, d_exponent(P.c0)), 0.0f, 0.0f, 1.0f};   // (the last row of an odd system)
    else if (!(s0.ok && s1.ok && row_fits(top))) D = block_of(P, i0, n).D;
    return minv(D);
}

template <bool RG>
__device__ __forceinline__ PrepRow prep_row(const MpArgs& p, int64_t j, int64_t k, Keep keep = Keep::normal)
{
    const PairRow P = load_pair<RG>(p, j, 2 * k, keep);
    const int64_t i0 = 2 * k;
    PrepRow r = prep_of(i0 >= 2 && i0 + 3 < p.n ? block_inner(P, i0, p.n) : block_of(P, i0, p.n));
    r.y = make_double2(P.y0, i0 + 1 < p.n ? P.y1 : 0.0);
    return r;
}

// A run of block rows of one system whose band slots all lie inside it
// (contiguous rows, every pair 16-byte aligned): the arrays from the run's
// first row on, a null outer band zero.  One address per array and run instead
// of the general row's index arithmetic and tests.
struct PairRun { const double *a, *b, *c, *d, *e, *y; };

__device__ __forceinline__ PairRun pair_run(const MpArgs& p, int64_t row)
{
    return {p.a ? p.a + row : nullptr, p.b + row, p.c + row, p.d + row, p.e ? p.e + row : nullptr, p.y + row};
}

__device__ __forceinline__ PairRow load_run(const PairRun& s, int k, Keep keep, uint64_t pol)
{
    const double2 z = make_double2(0.0, 0.0);
    const double2 a = s.a ? ldg2(s.a + 2 * k, keep, pol) : z;
    const double2 b = ldg2(s.b + 2 * k, keep, pol), c = ldg2(s.c + 2 * k, keep, pol);
    const double2 d = ldg2(s.d + 2 * k, keep, pol);
    const double2 e = s.e ? ldg2(s.e + 2 * k, keep, pol) : z;
    const double2 y = ldg2(s.y + 2 * k, keep, pol);
    return {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, e.x, e.y, y.x, y.y};
}

// r = y - A x of a block row whose band slots all lie inside the system
// (x_{i0-2..i0+3} = xm, xc, xp; the FMA order of residual_kernel), row-scaled
// and normalised by its diagonal block's inverse (formed again: cheaper than
// keeping it): the next right-hand side.
__device__ __forceinline__ float2 residual_inner(const PairRow& P, bool has_a, bool has_e, double2 xm, double2 xc,
                                                 double2 xp, int64_t i0, int64_t n)
{
    double r0 = fma(-P.c0, xc.x, P.y0), r1 = fma(-P.c1, xc.y, P.y1);
    if (has_a) { r0 = fma(-P.a0, xm.x, r0); r1 = fma(-P.a1, xm.y, r1); }
    r0 = fma(-P.b0, xm.y, r0); r1 = fma(-P.b1, xc.x, r1);
    r0 = fma(-P.d0, xc.y, r0); r1 = fma(-P.d1, xp.x, r1);
    if (has_e) { r0 = fma(-P.e0, xp.x, r0); r1 = fma(-P.e1, xp.y, r1); }
    const RowScale s0 = row_scale(P.c0), s1 = row_scale(P.c1);
    int top = 0;
    M2 D = {d2f_row(P.c0, s0, top), d2f_row(P.d0, s0, top), d2f_row(P.b1, s1, top), d2f_row(P.c1, s1, top)};
    float f0 = d2f_row(r0, s0, top), f1 = d2f_row(r1, s1, top);
    if (!(s0.ok && s1.ok && row_fits(top))) {
        D = block_of(P, i0, n).D;
        f0 = d2f_scaled(r0, d_exponent(P.c0)); f1 = d2f_scaled(r1, d_exponent(P.c1));
    }
    const M2 Mi = minv(D);
    return make_float2(fmaf(Mi.m0, f0, Mi.m1 * f1), fmaf(Mi.m2, f0, Mi.m3 * f1));
}

// Rows i0 = 2k, i0 + 1 of the rhs of system j (loaded by prep_row) -> the
// contiguous copy Yc, one 16-byte store where the pair is aligned.
__device__ __forceinline__ void store_rhs_pair(const MpArgs& p, int64_t j, int64_t i0, double2 y)
{
    const int64_t q = j * p.n + i0;
    if (i0 + 1 < p.n) {
        if ((q & 1) == 0) *reinterpret_cast<double2*>(p.Yc + q) = y;   // (Yc is 256-byte aligned)
        else { p.Yc[q] = y.x; p.Yc[q + 1] = y.y; }
    } else {
        p.Yc[q] = y.x;
    }
}

__device__ __forceinline__ void prep_store(const MpArgs& p, int64_t q, const PrepRow& r)
{
    // (the rhs copy Yc is written by the callers, which have y in hand)
    p.S0[2 * q] = make_float4(r.L.m0, r.L.m1, r.L.m2, r.L.m3);
    p.S0[2 * q + 1] = make_float4(r.U.m0, r.U.m1, r.U.m2, r.U.m3);
}

// per-system flags and norms of a solve
__global__ void __launch_bounds__(kMpThreads)
mp_init_kernel(MpArgs p)
{
    pdl_wait();
    pdl_release();
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, st = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = t0; j < p.m; j += st) { p.fin[j] = 0; p.status[j] = 0; p.est[j] = 0.0f; p.fail[j] = 0; }
    for (int64_t q = t0; q < (int64_t)kMpMaxPasses * p.m; q += st) p.trunc[q] = 0u;
    for (int64_t q = t0; q < (int64_t)(p.max_sweeps + 1) * p.m; q += st) { p.ndx[q] = 0u; p.nx[q] = 0u; }
    for (int64_t q = t0; q < (int64_t)p.max_sweeps * kMpMaxPasses * p.m; q += st) p.ndx_pre[q] = 0u;
    if (t0 == 0) { *p.nfail = 0; if (p.ctr) *p.ctr = 0; }
    for (int64_t q = t0; q <= p.max_sweeps; q += st) p.live[q] = (int)p.m;
    for (int64_t q = t0; q < 2 * p.m; q += st) p.dnorm[q] = 0u;
    if (t0 == 0 && p.err) *p.err = 0;
}

template <bool RG>
__global__ void __launch_bounds__(kMpThreads)
mp_prep_kernel(MpArgs p)
{
    pdl_wait();
    const int64_t nb = (p.n + 1) / 2;
    const int64_t total = p.m * nb;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = q / nb, k = q - j * nb;
        const PrepRow r = prep_row<RG>(p, j, k);
        prep_store(p, q, r);
        p.R[0][q] = r.Y;
        store_rhs_pair(p, j, 2 * k, r.y);
    }
    pdl_release();                                // (multi-wave grid: release once this CTA is done)
}

// The first right-hand side of the systems the windowed sweep 0 leaves to the
// general passes (the windows keep theirs in shared memory; 4 bytes per row
// that no other system's solve would read).
template <bool RG>
__global__ void __launch_bounds__(kMpThreads)
mp_rhs_kernel(MpArgs p, cudaGraphConditionalHandle windows, cudaGraphConditionalHandle full, bool gate)
{
    pdl_wait();
    pdl_release();                                // one wave of persistent CTAs: the successor may queue now
    const bool left = __ldg(p.nfail) != 0;
    if (gate && blockIdx.x == 0 && threadIdx.x == 0) {
        // no system left: the sweeps go on with sweep 1 (sweep 0 takes no
        // decision when more than one may run, and they are two at least)
        *p.ctr = left ? 0 : 1;
        cudaGraphSetConditional(windows, left ? 0u : 1u);
        cudaGraphSetConditional(full, left ? 1u : 0u);
    }
    if (!left) return;
    const int64_t nb = (p.n + 1) / 2;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < p.m * nb; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = q / nb;
        if (__ldg(p.fail + j)) p.R[0][q] = prep_row<RG>(p, j, q - j * nb).Y;
    }
}

// ---------------------------------------------------------------------------
// FP32 block PCR pass (windows + halos at block level G, or whole subsystems)
// ---------------------------------------------------------------------------
// One window of a global FP32 block-PCR pass (K strides at level G, halo H).
// Each thread keeps the rows it owns (k = tid + q*blockDim) in registers;
// shared memory holds one copy of the level's rows (L and U as float4 arrays,
// Y as float2), read for the two neighbours of a row and rewritten after
// every stride: 80 bytes read and 40 written per row and stride.
template <int RPT>
__device__ __forceinline__ void mp_pass_item(const MpPassArgs& p, int64_t j, int64_t r, int64_t w,
                                             float4* sL, float4* sU, float2* sY, unsigned* s_max)
{
    const int64_t nb = p.nb;
    if (r >= nb) return;
    const int64_t nr = (nb - 1 - r) / p.G + 1;
    const int64_t wlo = w * (int64_t)p.L;
    if (wlo >= nr) return;
    const int64_t whi = min(wlo + (int64_t)p.L, nr);
    const int64_t t0 = max(wlo - (int64_t)p.H, (int64_t)0);
    const int64_t t1 = min(whi + (int64_t)p.H, nr);
    const int TR = (int)(t1 - t0);
    const int tid = threadIdx.x, bd = blockDim.x;
    const int64_t g0 = j * nb + r;                 // block row of local t = 0
    const int K = p.K;

    M2 Lr[RPT], Ur[RPT];
    float2 Yr[RPT];
#pragma unroll
    for (int q = 0; q < RPT; q++) {
        const int k = tid + q * bd;
        Lr[q] = {0.0f, 0.0f, 0.0f, 0.0f}; Ur[q] = Lr[q]; Yr[q] = make_float2(0.0f, 0.0f);
        if (k < TR) {
            const int64_t gi = g0 + (t0 + k) * p.G;
            const float4 lv = p.srcLU[2 * gi], uv = p.srcLU[2 * gi + 1];
            const float2 yv = p.srcY[gi];
            sL[k] = lv; sU[k] = uv; sY[k] = yv;
            Lr[q] = m2(lv); Ur[q] = m2(uv); Yr[q] = yv;
        }
    }
    if (tid == 0) s_max[0] = 0u;
    __syncthreads();

    for (int st = 0; st < K; st++) {
        const int dl = 1 << st;
        // rows this stride must produce: the window widened by the halo the
        // remaining strides of the pass still consume
        const int64_t rem = (int64_t(1) << K) - (int64_t(2) << st);   // block halo = 2^K - 1
        const int klo = (int)(max(wlo - rem, (int64_t)0) - t0);
        const int khi = (int)(min(whi + rem, nr) - t0);
        // A row without a neighbour at distance dl has exactly zero coupling
        // towards it (the boundary blocks are zero at level 0 and stay zero),
        // so the neighbour index is clamped into the tile instead of
        // branching: the clamped row is finite and enters multiplied by zero.
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const int k = tid + q * bd;
            if (k >= klo && k < khi) {
                const int km = max(k - dl, 0), kp = min(k + dl, TR - 1);
                M2 Mi;
                reduce_row(Lr[q], Ur[q], Yr[q], m2(sL[km]), m2(sU[km]), sY[km], m2(sL[kp]), m2(sU[kp]), sY[kp],
                           Lr[q], Ur[q], Yr[q], Mi);
            }
        }
        __syncthreads();                                   // every read of this stride is done
        if (st == K - 1) break;
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const int k = tid + q * bd;
            if (k >= klo && k < khi) { sL[k] = f4(Lr[q]); sU[k] = f4(Ur[q]); sY[k] = Yr[q]; }
        }
        __syncthreads();
    }

    float lmax = 0.0f;
#pragma unroll
    for (int q = 0; q < RPT; q++) {
        const int k = tid + q * bd;
        const int64_t t = t0 + k;
        if (k < TR && t >= wlo && t < whi) {
            const int64_t gi = g0 + t * p.G;
            p.dstLU[2 * gi] = f4(Lr[q]);
            p.dstLU[2 * gi + 1] = f4(Ur[q]);
            p.dstY[gi] = Yr[q];
            lmax = fmaxf(lmax, fmaxf(amaxm(Lr[q]), amaxm(Ur[q])));
        }
    }
    lmax = warp_max(lmax);
    if ((tid & 31) == 0) {
        atomic_max_pos(&p.trunc_out[j], lmax);
        atomic_max_pos(&s_max[0], lmax);
    }
    __syncthreads();
    // A window whose couplings all vanished is decoupled: its rows already
    // hold X = Y.  Write them now; if every window of the system is
    // decoupled the later passes of this sweep skip the system.
    if (__uint_as_float(s_max[0]) < kTrunc) {
        float xm = 0.0f;
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const int k = tid + q * bd;
            const int64_t t = t0 + k;
            if (k < TR && t >= wlo && t < whi) {
                const int64_t i0 = 2 * (r + t * p.G);
                p.dx[j * p.n + i0] = Yr[q].x;
                xm = fmaxf(xm, fabsf(Yr[q].x));
                if (i0 + 1 < p.n) { p.dx[j * p.n + i0 + 1] = Yr[q].y; xm = fmaxf(xm, fabsf(Yr[q].y)); }
            }
        }
        xm = warp_max(xm);
        if ((tid & 31) == 0) atomic_max_pos(&p.ndx_pre_out[j], xm);
    }
}

// Loads rows [t0, t0 + TR) of subsystem r (level G) of system j into the
// swizzled tile.
__device__ __forceinline__ void cr_load(const MpPassArgs& p, int64_t j, int64_t r, int64_t t0, int TR,
                                        float4* sL, float4* sU, float2* sY)
{
    const int64_t g0 = j * p.nb + r;
    for (int k = threadIdx.x; k < TR; k += blockDim.x) {
        const int64_t gi = g0 + (t0 + k) * p.G;
        const int s = swz(k);
        sL[s] = p.srcLU[2 * gi]; sU[s] = p.srcLU[2 * gi + 1]; sY[swzy(k)] = p.srcY[gi];
    }
    __syncthreads();
}

// dx rows of tile rows [klo, khi) (tile row k = subsystem row t0 + k of
// subsystem r at level G) and their |dx| maximum into *norm.
__device__ __forceinline__ void cr_store(const MpPassArgs& p, int64_t j, int64_t r, int64_t t0, int klo, int khi,
                                         const float2* sY, unsigned* norm)
{
    float xmx = 0.0f;
    for (int k = klo + threadIdx.x; k < khi; k += blockDim.x) {
        const int64_t i0 = 2 * (r + (t0 + k) * p.G);      // first row of the block row
        const float2 xv = sY[swzy(k)];
        p.dx[j * p.n + i0] = xv.x;
        xmx = fmaxf(xmx, fabsf(xv.x));
        if (i0 + 1 < p.n) { p.dx[j * p.n + i0 + 1] = xv.y; xmx = fmaxf(xmx, fabsf(xv.y)); }
    }
    xmx = warp_max(xmx);
    if ((threadIdx.x & 31) == 0) atomic_max_pos(norm, xmx);
}

// A whole subsystem (nr <= TRmax rows at level G) by block cyclic reduction
// to the top (or until truncation) and back substitution: about 2 row
// updates per row instead of log2(nr).
__device__ __forceinline__ void mp_final_item(const MpPassArgs& p, int64_t j, int64_t r,
                                              float4* sL, float4* sU, float2* sY)
{
    if (r >= p.nb) return;
    const int nr = (int)((p.nb - 1 - r) / p.G + 1);
    cr_load(p, j, r, 0, nr, sL, sU, sY);
    const int top = cr_reduce(sL, sU, sY, nr, 31, 0, nr);   // never -1 on a whole subsystem
    cr_substitute(sL, sU, sY, nr, top);
    cr_store(p, j, r, 0, 0, nr, sY, &p.ndx[(int64_t)p.sweep * p.m + j]);
}

// Windowed truncated cyclic reduction at level 0 (the first pass of a large
// system): window [wlo, wlo + L) with a halo of H = 2^(K+1) rows each side.
// After l <= K levels the reduced rows the window depends on lie within
// 2^l - 1 rows of it and are exact when their own dependence (2^l - 1 rows
// further) is inside the tile; if they are decoupled, back substitution
// gives the window's dx with no other window involved.  Otherwise the system
// is marked for the general passes (block PCR windows + shared-memory
// finish) and the window writes nothing.
struct TryTile {
    int64_t j, wlo, whi, t0;
    int TR;
    bool whole;                                   // the tile holds the whole system
};

__device__ __forceinline__ TryTile try_tile(const MpPassArgs& p, int64_t item, int64_t j)
{
    TryTile t;
    t.j = j;
    const int64_t w = item - t.j * p.nwin;
    t.wlo = w * (int64_t)p.L;
    t.whi = min(t.wlo + (int64_t)p.L, p.nb);
    t.t0 = max(t.wlo - (int64_t)p.H, (int64_t)0);
    const int64_t t1 = min(t.whi + (int64_t)p.H, p.nb);
    t.TR = (int)(t1 - t.t0);
    t.whole = t.t0 == 0 && t1 == p.nb;
    return t;
}

// next item of this CTA with work: running system, window inside it, and
// (after sweep 0) a system the windowed pass solves
__device__ __forceinline__ int64_t try_next(const MpPassArgs& p, int64_t item, int64_t items, int64_t& j)
{
    for (; item < items; item += gridDim.x) {
        j = item / p.nwin;
        if (__ldg(p.fin + j)) continue;
        if (p.sweep > 0 && __ldg(p.fail + j)) continue;
        if ((item - j * p.nwin) * (int64_t)p.L >= p.nb) continue;
        break;
    }
    return item;
}

__device__ __forceinline__ void try_solve(const MpPassArgs& p, const TryTile& t, float4* sL, float4* sU, float2* sY)
{
    cr_load(p, t.j, 0, t.t0, t.TR, sL, sU, sY);
    // a tile holding the whole system needs no truncation: reduce to the top
    const int kmax = t.whole ? 31 : p.K;
    const int top = cr_reduce(sL, sU, sY, t.TR, kmax, (int)(t.wlo - t.t0), (int)(t.whi - t.t0));
    if (top < 0) {
        if (threadIdx.x == 0 && atomicOr(&p.fail[t.j], 1) == 0) atomicAdd(p.nfail, 1);
        return;
    }
    // x_s = x_{s-1} + dx_s on the window's rows, straight from the tile.  The
    // norms go straight into the sweep's: if another window of the system
    // fails, the general passes redo these rows with values equal to within
    // the truncation, so the maxima stand either way.
    const int klo = (int)(t.wlo - t.t0), khi = (int)(t.whi - t.t0);
    const XView xv = x_view(p.sweep, p.max_sweeps, p.X0f, p.xout, p.oss, p.ors, p.rg);
    // sweep 1 of a contiguous batch with aligned pairs: one address per array
    // and tile, and x_0 on its way from memory during the substitution (the
    // last row of an odd system goes the general way below)
    const float* __restrict__ xs = xv.srcf + t.j * p.n + 2 * t.t0;
    double* __restrict__ xd = xv.dst + t.j * xv.dss + 2 * t.t0;
    const bool run = xv.srcf && !xv.drg && xv.drs == 1 &&
                     ((reinterpret_cast<uintptr_t>(xs) & 7) | (reinterpret_cast<uintptr_t>(xd) & 15)) == 0;
    const int done = run ? (int)(min(t.whi, p.n / 2) - t.t0) : klo;
    float2 x0[kMpTryRows / kMpTryThreads];
#pragma unroll
    for (int u = 0; u < kMpTryRows / kMpTryThreads; u++) {
        const int k = klo + (int)threadIdx.x + u * kMpTryThreads;
        if (k < done) x0[u] = reinterpret_cast<const float2*>(xs)[k];
    }
    cr_substitute(sL, sU, sY, t.TR, top);
    float dmax = 0.0f;
    unsigned long long xbits = 0ull;
#pragma unroll
    for (int u = 0; u < kMpTryRows / kMpTryThreads; u++) {
        const int k = klo + (int)threadIdx.x + u * kMpTryThreads;
        if (k < done) {
            const float2 d = sY[swzy(k)];
            const double2 x = make_double2(__dadd_rn(f2d(x0[u].x), f2d(d.x)), __dadd_rn(f2d(x0[u].y), f2d(d.y)));
            reinterpret_cast<double2*>(xd)[k] = x;
            dmax = fmaxf(dmax, fmaxf(fabsf(d.x), fabsf(d.y)));
            xbits = max(xbits, max(absbits(x.x), absbits(x.y)));
        }
    }
    for (int k = done + (int)threadIdx.x; k < khi; k += blockDim.x) {
        const int64_t i0 = 2 * (t.t0 + k);
        const float2 v = sY[swzy(k)];
        x_update(xv, p.n, t.j, i0, v.x, dmax, xbits);
        if (i0 + 1 < p.n) x_update(xv, p.n, t.j, i0 + 1, v.y, dmax, xbits);
    }
    dmax = warp_max(dmax);
    const float xmax = warp_max(d2f_scaled(__longlong_as_double((long long)xbits), 0));
    if ((threadIdx.x & 31) == 0) {
        atomic_max_pos(&p.ndx[(int64_t)p.sweep * p.m + t.j], dmax);
        atomic_max_pos(&p.nx[t.j], xmax);
    }
}

// Persistent CTAs over the windows, 4 per SM (40 KB tiles of 1024 rows, at
// most 64 registers): the reduction levels are short dependent chains
// separated by barriers, so several tiles per SM keep it busy (5 per SM at
// 48 registers measured 1 % slower on GB300, 6 at 40 no faster).
__global__ void __launch_bounds__(kMpTryThreads, 4)
mp_try_kernel(MpPassArgs p)
{
    extern __shared__ float4 fsm[];
    pdl_wait();
    pdl_release();                                // one wave of persistent CTAs: the successor may queue now
    mp_resolve(p);
    if (p.skip0 && p.sweep == 0) return;          // sweep 0 ran in the fused kernel
    if (__ldg(p.live) == 0) return;               // every system finished in an earlier sweep
    const int TRs = mp_pass_rows(p.TRmax);
    float4* sL = fsm;
    float4* sU = fsm + TRs;
    float2* sY = reinterpret_cast<float2*>(fsm + 2 * TRs);
    const int64_t items = p.m * p.nwin;
    int64_t j = 0;
    for (int64_t it = try_next(p, blockIdx.x, items, j); it < items; it = try_next(p, it + gridDim.x, items, j)) {
        try_solve(p, try_tile(p, it, j), sL, sU, sY);
        __syncthreads();
    }
}

// Sweep 0 fused (prep, windowed cyclic reduction and the first refinement),
// for windows that decouple (or hold the whole system).  Per window tile:
//  1. FP64 bands and y of the tile's block rows -> row-scaled, normalised FP32
//     blocks in shared memory; the window's own rows also go to S0 for the
//     later sweeps and the general passes;
//  2. cyclic reduction and back substitution (as mp_try_item): dx_0;
//  3. x_0 = dx_0 on the window's rows and one block row each side (exact
//     there: the valid region of the tile reaches 2 block rows beyond the
//     window), written to X0f; norms of dx_0 and x_0;
//  4. r_0 = y - A x_0 in FP64 for the window's rows (bands and y read again,
//     from L2), row-scaled and normalised -> R[1].
// No decision is needed in sweep 0, so nothing waits for other windows.  A
// window whose system stays coupled marks it and stops after step 1; the
// general passes and the refinement kernel then take the whole system.
// (steps 1 and 4 of an inner tile)
__device__ __forceinline__ void first_prep(const MpArgs& p, const PairRun& run, int64_t j, int64_t t0, int TR, int klo,
                                           int khi, float4* sL, float4* sU, float2* sY)
{
    const int64_t nb = (p.n + 1) / 2;
    float4* __restrict__ S0 = p.S0 + 2 * (j * nb + t0);
    double* __restrict__ Yc = p.Yc + j * p.n + 2 * t0;
    const uint64_t pol = tma::policy_evict_last();
    for (int k = threadIdx.x; k < TR; k += blockDim.x) {
        const PairRow P = load_run(run, k, Keep::last, pol);
        const PrepRow r = prep_of(block_inner(P, 2 * (t0 + k), p.n));
        const int sk = swz(k);
        sL[sk] = f4(r.L); sU[sk] = f4(r.U); sY[swzy(k)] = r.Y;
        if (k >= klo && k < khi) {
            S0[2 * k] = f4(r.L);
            S0[2 * k + 1] = f4(r.U);
            *reinterpret_cast<double2*>(Yc + 2 * k) = make_double2(P.y0, P.y1);
        }
    }
}

__device__ __forceinline__ void first_residual(const MpArgs& p, const PairRun& run, int64_t j, int64_t t0, int klo,
                                               int khi, const double2* sX)
{
    float2* __restrict__ R = p.R[1] + j * ((p.n + 1) / 2) + t0;
    const uint64_t pol = tma::policy_evict_first();
    for (int k = klo + (int)threadIdx.x; k < khi; k += blockDim.x) {
        const PairRow P = load_run(run, k, Keep::first, pol);
        R[k] = residual_inner(P, run.a != nullptr, run.e != nullptr, sX[k - 1], sX[k], sX[k + 1], 2 * (t0 + k), p.n);
    }
}

template <bool RG>
__device__ __forceinline__ void first_item(const MpArgs& p, const MpWindows& g, int64_t item, int64_t j,
                                           float4* sL, float4* sU, float2* sY)
{
    const int tid = threadIdx.x, bd = blockDim.x;
    const int64_t n = p.n, nb = (n + 1) / 2;
    const int64_t w = item - j * g.nwin;
    const int64_t wlo = w * (int64_t)g.L, whi = min(wlo + (int64_t)g.L, nb);
    const int64_t t0 = max(wlo - (int64_t)g.H, (int64_t)0), t1 = min(whi + (int64_t)g.H, nb);
    const int TR = (int)(t1 - t0);
    const bool whole = t0 == 0 && t1 == nb;

    // an inner tile: one aligned run of rows, every band slot in the system
    int64_t base = j * p.ss, nj = n;
    if (RG) { const longlong2 r = __ldg(p.rg + j); base = r.x; nj = r.y; }
    const bool inner = (RG || p.rs == 1) && t0 >= 1 && 2 * t1 + 2 <= nj && p.vec && ((base | (j * n)) & 1) == 0;
    if (inner) first_prep(p, pair_run(p, base + 2 * t0), j, t0, TR, (int)(wlo - t0), (int)(whi - t0), sL, sU, sY);
    else for (int k = tid; k < TR; k += bd) {
        const int64_t kb = t0 + k;
        const PrepRow r = prep_row<RG>(p, j, kb, Keep::last);
        const int sk = swz(k);
        sL[sk] = f4(r.L); sU[sk] = f4(r.U); sY[swzy(k)] = r.Y;
        if (kb >= wlo && kb < whi) {
            prep_store(p, j * nb + kb, r);
            store_rhs_pair(p, j, 2 * kb, r.y);
        }
    }
    __syncthreads();
    const int klo = (int)(wlo - t0), khi = (int)(whi - t0);
    const int top = cr_reduce(sL, sU, sY, TR, whole ? 31 : g.K, klo, khi);
    if (top < 0) {
        if (tid == 0 && atomicOr(&p.fail[j], 1) == 0) atomicAdd(p.nfail, 1);
        return;
    }
    cr_substitute(sL, sU, sY, TR, top);           // ends with a barrier: the L slots are free

    // x_0 pairs, kept as double2 in the L slots for the residual's neighbours
    double2* sX = reinterpret_cast<double2*>(sL);
    const int xlo = max(klo - 1, 0), xhi = min(khi + 1, TR);
    float* __restrict__ X0 = p.X0f + j * n + 2 * t0;
    const bool even = ((j * n) & 1) == 0;
    const int pairs = (int)(n / 2 - t0);          // block rows of two rows
    float dmax = 0.0f;
    bool nan = false;
    for (int k = xlo + tid; k < xhi; k += bd) {
        const float2 v = sY[swzy(k)];
        sX[k] = make_double2(f2d(v.x), f2d(v.y));
        if (k >= klo && k < khi) {
            // x_0 = dx_0: one maximum for both norms
            const bool two = k < pairs;
            if (two && even) *reinterpret_cast<float2*>(X0 + 2 * k) = v;      // (X0f is 256-byte aligned)
            else { X0[2 * k] = v.x; if (two) X0[2 * k + 1] = v.y; }
            dmax = fmaxf(dmax, fabsf(v.x));
            nan |= v.x != v.x;
            if (two) { dmax = fmaxf(dmax, fabsf(v.y)); nan |= v.y != v.y; }
        }
    }
    const float xmax = warp_max(nan ? __int_as_float(0x7FC00000) : dmax);
    dmax = warp_max(dmax);
    if ((tid & 31) == 0) {
        atomic_max_pos(&p.ndx[j], dmax);
        atomic_max_pos(&p.nx[j], xmax);
    }
    __syncthreads();

    // r_0 = y - A x_0 on the window's block rows (FP64, same FMA order as the
    // refinement kernel), row-scaled and normalised -> the rhs of sweep 1
    if (inner) { first_residual(p, pair_run(p, base + 2 * t0), j, t0, klo, khi, sX); return; }
    for (int k = klo + tid; k < khi; k += bd) {
        const int64_t kb = t0 + k, i0 = 2 * kb;
        const PairRow P = load_pair<RG>(p, j, i0, Keep::first);
        const double2 xm = k > 0 ? sX[k - 1] : make_double2(0.0, 0.0);
        const double2 xc = sX[k];
        const double2 xp = k + 1 < TR ? sX[k + 1] : make_double2(0.0, 0.0);
        double r0 = P.y0;                          // row i0: x_{i0-2..i0+2} = xm.x xm.y xc.x xc.y xp.x
        r0 = fma(-P.c0, xc.x, r0);
        if (p.a && i0 >= 2) r0 = fma(-P.a0, xm.x, r0);
        if (i0 >= 1) r0 = fma(-P.b0, xm.y, r0);
        if (i0 + 1 < n) r0 = fma(-P.d0, xc.y, r0);
        if (p.e && i0 + 2 < n) r0 = fma(-P.e0, xp.x, r0);
        float rf1 = 0.0f;                          // row i0+1 (the identity row of an odd system: 0)
        if (i0 + 1 < n) {
            const int64_t i1 = i0 + 1;             // x_{i1-2..i1+2} = xm.y xc.x xc.y xp.x xp.y
            double r1 = P.y1;
            r1 = fma(-P.c1, xc.y, r1);
            if (p.a && i1 >= 2) r1 = fma(-P.a1, xm.y, r1);
            r1 = fma(-P.b1, xc.x, r1);
            if (i1 + 1 < n) r1 = fma(-P.d1, xp.x, r1);
            if (p.e && i1 + 2 < n) r1 = fma(-P.e1, xp.y, r1);
            rf1 = d2f_scaled(r1, d_exponent(P.c1));
        }
        const float rf0 = d2f_scaled(r0, d_exponent(P.c0));
        const M2 Mi = diag_inverse(P, i0, n);     // (formed again: cheaper than keeping it)
        p.R[1][j * nb + kb] = make_float2(fmaf(Mi.m0, rf0, Mi.m1 * rf1), fmaf(Mi.m2, rf0, Mi.m3 * rf1));
    }
}

// Persistent CTAs over the windows of all systems (40 KB tiles of 1024
// block rows, or whole systems of up to 2048), 4 per SM at most.
template <bool RG>
__global__ void __launch_bounds__(kMpTryThreads, 4)
mp_first_kernel(MpArgs p, MpWindows g)
{
    extern __shared__ float4 fsm[];
    pdl_wait();
    pdl_release();                                // one wave of persistent CTAs: the successor may queue now
    const int TRs = mp_pass_rows(g.TRmax);
    float4* sL = fsm;
    float4* sU = fsm + TRs;
    float2* sY = reinterpret_cast<float2*>(fsm + 2 * TRs);
    if (__ldg(p.live) == 0) return;               // the fused first sweeps finished every system
    const int64_t items = p.m * g.nwin;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int64_t j = it / g.nwin;
        if (__ldg(p.fin + j)) continue;           // finished by the fused first sweeps
        first_item<RG>(p, g, it, j, sL, sU, sY);
        __syncthreads();
    }
}

// 4 CTAs per SM up to 4 rows per thread (64 registers, 40 KB of shared
// memory each at 1024 block rows), 2 beyond
template <int RPT>
__global__ void __launch_bounds__(kMpThreads, RPT >= 8 ? 2 : 4)
mp_pass_kernel(MpPassArgs p)
{
    extern __shared__ float4 fsm[];
    __shared__ unsigned s_max[1];
    pdl_wait();
    pdl_release();                                // one wave of persistent CTAs: the successor may queue now
    mp_resolve(p);
    // the flags read here were written by earlier kernels: read-only cache
    if (__ldg(p.live) == 0) return;               // every system finished in an earlier sweep
    if (p.fail && __ldg(p.nfail) == 0) return;    // the windowed pass solved every system
    const int TRs = mp_pass_rows(p.TRmax);
    float4* sL = fsm;
    float4* sU = fsm + TRs;
    float2* sY = reinterpret_cast<float2*>(fsm + 2 * TRs);
    // grid-stride over the items (about one wave of CTAs)
    const int64_t items = p.m * p.G * p.nwin;
    for (int64_t blk = blockIdx.x; blk < items; blk += gridDim.x) {
        const int64_t item = blk / p.nwin;
        const int64_t w = blk - item * p.nwin;
        const int64_t j = item / p.G;
        const int64_t r = item - j * p.G;
        if (__ldg(p.fin + j)) continue;
        if (p.fail && !__ldg(p.fail + j)) continue;   // solved by the windowed cyclic-reduction pass
        if (p.trunc_in && __uint_as_float(__ldg(p.trunc_in + j)) < kTrunc) {
            // Every window of the previous pass found itself decoupled and
            // wrote its rows of dx (X = Y): item (0, 0) carries the |dx|
            // maximum they left into the sweep's norm, the rest is skipped.
            if (r == 0 && w == 0 && threadIdx.x == 0)
                atomicMax(&p.ndx[(int64_t)p.sweep * p.m + j], p.ndx_pre_in[j]);
            continue;
        }
        if (p.final_step) mp_final_item(p, j, r, sL, sU, sY);
        else mp_pass_item<RPT>(p, j, r, w, sL, sU, sY, s_max);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// refinement: x_s = x_{s-1} + dx_s (FP64), decide, r_s = y - A x_s
// ---------------------------------------------------------------------------
// Iterates: sweep 0 writes x_0 to X0f (workspace), every later sweep reads
// x_{s-1} and writes x_s in the output (the caller's y, or Xout when the
// report keeps y): a system that finishes in sweep s already holds its
// answer there, and the rhs is read from the copy Yc (x_view).

// Systems whose dx came from the general passes (all of them when no cyclic-
// reduction pass ran): x_s = x_{s-1} + dx_s and max |x_s|.
__global__ void __launch_bounds__(kMpThreads)
mp_xupdate_kernel(MpArgs p)
{
    __shared__ float s_red[kMpThreads / 32];
    pdl_wait();
    pdl_release();                                // one wave of persistent CTAs: the successor may queue now
    mp_resolve(p);
    const int s = p.sweep;
    if (__ldg(p.live + s) == 0) return;           // every system finished in an earlier sweep
    if (p.cr_mode && __ldg(p.nfail) == 0) return; // the cyclic-reduction passes updated every system
    const XView xv = x_view(s, p.max_sweeps, p.X0f, p.xout, p.oss, p.ors, p.rg);
    constexpr int XT = 4 * kMpThreads;            // rows per tile
    const int64_t n = p.n, tiles = (n + XT - 1) / XT;
    for (int64_t blk = blockIdx.x; blk < p.m * tiles; blk += gridDim.x) {
        const int64_t j = blk / tiles, t0 = (blk - j * tiles) * XT;
        if (__ldg(p.fin + j) != 0) continue;
        if (p.cr_mode && !__ldg(p.fail + j)) continue;
        float dmax = 0.0f;
        unsigned long long xbits = 0ull;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t i = t0 + threadIdx.x + u * kMpThreads;
            if (i < n) x_update(xv, n, j, i, p.dx[j * n + i], dmax, xbits);
        }
        float xmax = warp_max(d2f_scaled(__longlong_as_double((long long)xbits), 0));
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = xmax;
        __syncthreads();
        if (threadIdx.x == 0) {
            float v = 0.0f;
            for (int w = 0; w < kMpThreads / 32; w++) v = fmaxf(v, s_red[w]);
            atomic_max_pos(&p.nx[(int64_t)s * p.m + j], v);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ UpDecision up_decide(const MpArgs& p, int64_t j)
{
    const int s = p.sweep;
    if (s < 1) return stop_rule(s, 0.0f, 0.0f, 0.0f, p.tol, p.max_sweeps);
    return stop_rule(s, __uint_as_float(p.ndx[(int64_t)s * p.m + j]),
                     __uint_as_float(p.ndx[(int64_t)(s - 1) * p.m + j]),
                     __uint_as_float(p.nx[(int64_t)(s - 1) * p.m + j]), p.tol, p.max_sweeps);
}

// One thread per system: a system that is done (or out of sweeps) finishes in
// sweep s; its answer is already in the output.
__global__ void __launch_bounds__(kMpThreads)
mp_decide_kernel(MpArgs p)
{
    pdl_wait();
    pdl_release();
    mp_resolve(p);
    const int s = p.sweep;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    bool finish = false;
    if (j < p.m && p.fin[j] == 0) {
        const UpDecision D = up_decide(p, j);
        // A sweep without general passes takes the blocks of sweep 0, which
        // decoupled then, through the same reduction; should a window differ
        // all the same, its system stops here and is not called converged.
        const bool lost = p.windows_only && __ldg(p.fail + j) != 0;
        if (D.last || lost) {
            p.est[j] = lost ? __uint_as_float(0x7F800000u) : D.est;
            p.status[j] = D.done && !lost ? 1 : 2;    // 2: stopped at max_sweeps
            p.fin[j] = s + 1;
            finish = true;
        }
    }
    const int cnt = __syncthreads_count(finish);
    if (threadIdx.x == 0 && cnt > 0)
        for (int s2 = s + 1; s2 <= p.max_sweeps; s2++) atomicSub(&p.live[s2], cnt);
}

// Systems that fit one shared-memory tile (every block row of a system in
// one CTA): all sweeps of a system run inside its CTA, so nothing waits for
// the rest of the batch between sweeps and the whole solve is one launch.
// Per system:
//  1. FP64 bands and y -> row-scaled, normalised FP32 blocks in shared memory;
//  2. per sweep: cyclic reduction to the top (sweep 0, which keeps the factors
//     of its steps; later sweeps replay them on their rhs) and back
//     substitution (dx_s), x_s = x_{s-1} + dx_s in FP64, the maxima of |dx_s|
//     and |x_s| over the CTA, the stopping rule; if another sweep follows,
//     r_s = y - A x_s in FP64, row-scaled and normalised into the tile's rhs;
//  3. x -> the output, status, sweeps and estimate.
// y keeps the rhs until the final copy, so no copy of it is needed.
//
// Bound by latency: two CTAs of 512 threads fill an SM's registers at n=4096
// (FP64 pipe 41 %, ALU 45 %, issue 51 %; L2 and barrier waits).  Measured:
// reducing the matrix again in every sweep, from a copy of the blocks, m=4096
// n=4096 ADI 931 us; the factors kept instead, zero outer bands skipped and
// the tile's cheaper swizzles 870 (same bits).  Keeping the diagonal inverses
// as well costs more L2 traffic than the instructions it saves (+5 %), the
// factors in shared memory as generic addresses +3 %; the iterate as 16-byte
// pairs changes nothing.
__device__ __forceinline__ void block_max(unsigned& dmb, unsigned long long& xb, unsigned* red_d,
                                          unsigned long long* red_x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dmb = max(dmb, __shfl_xor_sync(0xffffffffu, dmb, o));
        xb = max(xb, __shfl_xor_sync(0xffffffffu, xb, o));
    }
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) { red_d[w] = dmb; red_x[w] = xb; }
    __syncthreads();
    dmb = 0u; xb = 0ull;
    for (int k = 0; k < nw; k++) { dmb = max(dmb, red_d[k]); xb = max(xb, red_x[k]); }
    __syncthreads();                              // the scratch is reused by the next call
}

constexpr int kMpNarrow = 256;                   // block rows of a system solved by 128 threads
constexpr int kMpSmallThreadsMax = 512;          // systems of >= 1024 block rows: 512 threads

// kKeep: sweep 0 keeps the factors of the reduction and later sweeps replay
// it; else they reduce a copy of the level-0 blocks again (launch_mp_small)
template <bool RG, bool kKeep>
__global__ void __launch_bounds__(kMpSmallThreadsMax, 2)
mp_small_kernel(MpArgs p)
{
    extern __shared__ float4 fsm[];
    __shared__ unsigned red_d[kMpSmallThreadsMax / 32];
    __shared__ unsigned long long red_x[kMpSmallThreadsMax / 32];
    __shared__ float4 s_last[3 * kCrLevels];
    pdl_wait();
    pdl_release();
    const int64_t n = p.n, nb = (n + 1) / 2;
    const int TR = (int)nb, TRs = mp_pass_rows(TR);
    float4* sL = fsm;
    float4* sU = fsm + TRs;
    float2* sY = reinterpret_cast<float2*>(fsm + 2 * TRs);
    const int tid = threadIdx.x, bd = blockDim.x;
    // this CTA's part of the workspace, the same for every system it solves
    // (what it writes stays in L2): the iterate, and the factors (or the blocks)
    // in the memory of S0 and R[], which follow each other (48 bytes per block
    // row)
    double* __restrict__ X = p.X0 + blockIdx.x * n;
    const CrFactors F{p.S0 + 3 * nb * blockIdx.x, s_last};
    for (int64_t j = blockIdx.x; j < p.m; j += gridDim.x) {
        unsigned any_a = 0u, any_e = 0u;          // bits of the outer bands inside the system
        for (int k = tid; k < TR; k += bd) {
            const int64_t i0 = 2 * (int64_t)k;
            const PairRow P = load_pair<RG>(p, j, i0);
            const PrepRow r = prep_of(i0 >= 2 && i0 + 3 < n ? block_inner(P, i0, n) : block_of(P, i0, n));
            if (i0 >= 2) any_a |= magbits(P.a0) | magbits(P.a1);
            if (i0 + 2 < n) any_e |= magbits(P.e0);
            if (i0 + 3 < n) any_e |= magbits(P.e1);
            const int sk = swz(k);
            sL[sk] = f4(r.L); sU[sk] = f4(r.U); sY[swzy(k)] = r.Y;
            if (!kKeep) { F.g[2 * k] = f4(r.L); F.g[2 * k + 1] = f4(r.U); }
        }
        // an outer band that is zero in the whole system (one-sided operators)
        // is treated like a missing one: neither read nor multiplied again
        const bool has_a = __syncthreads_or(any_a != 0u), has_e = __syncthreads_or(any_e != 0u);
        float ndp = 0.0f, nxp = 0.0f;
        UpDecision D{false, false, 0.0f};
        int s = 0, top = 0;
        for (;; s++) {
            // (a whole system: never -1)
            if (!kKeep || s == 0) top = cr_reduce<kKeep>(sL, sU, sY, TR, 31, 0, TR, F);
            else cr_replay(F, sY, TR, top);
            cr_substitute(sL, sU, sY, TR, top);
            unsigned dmb = 0u;
            unsigned long long xb = 0ull;
            for (int k = tid; k < TR; k += bd) {
                const float2 v = sY[swzy(k)];
                const int64_t i0 = 2 * (int64_t)k;
                const double x0 = s ? __dadd_rn(X[i0], f2d(v.x)) : f2d(v.x);
                X[i0] = x0;
                dmb = max(dmb, __float_as_uint(fabsf(v.x)));
                xb = max(xb, absbits(x0));
                if (i0 + 1 < n) {
                    const double x1 = s ? __dadd_rn(X[i0 + 1], f2d(v.y)) : f2d(v.y);
                    X[i0 + 1] = x1;
                    dmb = max(dmb, __float_as_uint(fabsf(v.y)));
                    xb = max(xb, absbits(x1));
                }
            }
            block_max(dmb, xb, red_d, red_x);     // (its barriers also publish X to the CTA)
            // non-negative floats order like their bits, a nan above everything
            const float nd = __uint_as_float(dmb);
            const float nx = d2f_scaled(__longlong_as_double((long long)xb), 0);
            D = stop_rule(s, nd, ndp, nxp, p.tol, p.max_sweeps);
            if (D.last) break;
            ndp = nd; nxp = nx;
            for (int k = tid; k < TR; k += bd) {
                const int64_t i0 = 2 * (int64_t)k;
                const PairRow P = load_pair<RG>(p, j, i0, Keep::normal, has_a, has_e);
                const double xm2 = i0 >= 2 ? X[i0 - 2] : 0.0, xm1 = i0 >= 1 ? X[i0 - 1] : 0.0, x0 = X[i0];
                const double x1 = i0 + 1 < n ? X[i0 + 1] : 0.0, x2 = i0 + 2 < n ? X[i0 + 2] : 0.0;
                const double x3 = i0 + 3 < n ? X[i0 + 3] : 0.0;
                double r0 = fma(-P.c0, x0, P.y0);
                if (has_a && i0 >= 2) r0 = fma(-P.a0, xm2, r0);
                if (i0 >= 1) r0 = fma(-P.b0, xm1, r0);
                if (i0 + 1 < n) r0 = fma(-P.d0, x1, r0);
                if (has_e && i0 + 2 < n) r0 = fma(-P.e0, x2, r0);
                const float rf0 = d2f_scaled(r0, d_exponent(P.c0));
                float rf1 = 0.0f;                 // the identity row of an odd system's last block row
                if (i0 + 1 < n) {
                    double r1 = fma(-P.c1, x1, P.y1);
                    if (has_a && i0 >= 1) r1 = fma(-P.a1, xm1, r1);
                    r1 = fma(-P.b1, x0, r1);
                    if (i0 + 2 < n) r1 = fma(-P.d1, x2, r1);
                    if (has_e && i0 + 3 < n) r1 = fma(-P.e1, x3, r1);
                    rf1 = d2f_scaled(r1, d_exponent(P.c1));
                }
                const M2 Mi = diag_inverse(P, i0, n);
                sY[swzy(k)] = make_float2(fmaf(Mi.m0, rf0, Mi.m1 * rf1), fmaf(Mi.m2, rf0, Mi.m3 * rf1));
                if (!kKeep) {
                    const int sk = swz(k);
                    sL[sk] = F.g[2 * k]; sU[sk] = F.g[2 * k + 1];
                }
            }
            if (!kKeep) __syncthreads();
        }
        for (int64_t i = tid; i < n; i += bd) x_write(p.xout, p.oss, p.ors, RG ? p.rg : nullptr, j, i, X[i]);
        if (tid == 0) { p.fin[j] = s + 1; p.status[j] = D.done ? 1 : 2; p.est[j] = D.est; }
        __syncthreads();                          // the next system reuses the tile
    }
}

// r_s = y - A x_s (FP64, FMA chain) for the systems still running, row-scaled
// to FP32 by the power of two of the main diagonal; the odd row of a block
// row reaches the even lane by a shuffle, which normalises the pair by the
// block's diagonal inverse (formed again from the bands it has in hand) ->
// R[(s+1) & 1], the rhs of sweep s+1.
template <bool RG>
__device__ __forceinline__ void residual_tile(const MpArgs& p, int s, const XView& xv, int64_t j, int64_t tile,
                                              double* sx)
{
    const int tid = threadIdx.x;
    const int64_t n = p.n;
    constexpr int XR = kMpTile / kMpThreads;             // rows per thread
    const int64_t t0 = tile * kMpTile, t1 = min(t0 + kMpTile, n);
    const int64_t ih = tid < 2 ? t0 - 2 + tid : t1 + tid - 2;          // halo row of threads 0-3
    const bool halo = tid < 4 && ih >= 0 && ih < n;
    // the system's rows in the caller arrays (a ragged system ends at nj <= n:
    // identity rows beyond, and its slots coupling to them are zero)
    int64_t base = j * p.ss, rs = p.rs, nj = n;
    if (RG) { const longlong2 g = __ldg(p.rg + j); base = g.x; rs = 1; nj = g.y; }
    auto x_at = [&](int64_t i) {
        return xv.dstf ? f2d(xv.dstf[j * n + i]) : x_read(xv.dst, xv.dss, xv.drs, RG ? xv.drg : nullptr, j, i);
    };
    double ba[XR], bb[XR], bc[XR], bd[XR], be[XR], by[XR];
#pragma unroll
    for (int u = 0; u < XR; u++) {
        const int64_t i = t0 + tid + u * kMpThreads;
        ba[u] = 0.0; bb[u] = 0.0; bc[u] = 1.0; bd[u] = 0.0; be[u] = 0.0; by[u] = 0.0;
        if (i < t1) {
            if (i < nj) {
                const int64_t g = base + i * rs;
                ba[u] = p.a ? p.a[g] : 0.0; bb[u] = p.b[g]; bc[u] = p.c[g];
                if (i + 1 < nj) bd[u] = p.d[g];
                if (p.e && i + 2 < nj) be[u] = p.e[g];
            }
            by[u] = p.Yc[j * n + i];
            sx[tid + u * kMpThreads + 2] = x_at(i);
        }
    }
    if (halo) sx[ih - t0 + 2] = x_at(ih);
    __syncthreads();

    const int64_t nb = (n + 1) / 2;
    const bool interior = t0 >= 2 && t1 + 2 <= n;          // no band slot of the tile falls outside the system
#pragma unroll
    for (int u = 0; u < XR; u++) {
        const int r0 = tid + u * kMpThreads;               // row within the tile (even lanes: first row of a block row)
        const int64_t i = t0 + r0;
        const bool even = (r0 & 1) == 0;
        // the row's part of the diagonal block, scaled as in the prep (an
        // identity row past an odd system's end)
        const int sh = d_exponent(bc[u]);
        const bool in = i < t1;
        const float dc = in ? d2f_scaled(bc[u], sh) : 1.0f;
        const float dn = in && (!even || i + 1 < n) ? d2f_scaled(even ? bd[u] : bb[u], sh) : 0.0f;
        const float dc1 = __shfl_xor_sync(0xffffffffu, dc, 1), dn1 = __shfl_xor_sync(0xffffffffu, dn, 1);
        float rf = 0.0f;
        if (i < t1) {
            const int li = r0 + 2;
            double r = by[u];
            r = fma(-bc[u], sx[li], r);
            if (interior) {
                if (p.a) r = fma(-ba[u], sx[li - 2], r);
                r = fma(-bb[u], sx[li - 1], r);
                r = fma(-bd[u], sx[li + 1], r);
                if (p.e) r = fma(-be[u], sx[li + 2], r);
            } else {
                if (p.a && i >= 2) r = fma(-ba[u], sx[li - 2], r);
                if (i >= 1) r = fma(-bb[u], sx[li - 1], r);
                if (i + 1 < n) r = fma(-bd[u], sx[li + 1], r);
                if (p.e && i + 2 < n) r = fma(-be[u], sx[li + 2], r);
            }
            rf = d2f_scaled(r, sh);
        }
        // (the partner of row n-1 of an odd system is the identity row of the
        // padded block, r = 0: its lane lies past t1 and keeps rf = 0)
        const float rf1 = __shfl_xor_sync(0xffffffffu, rf, 1);
        if (even && in) {
            const M2 Mi = minv({dc, dn, dn1, dc1});
            p.R[(s + 1) & 1][j * nb + (i >> 1)] = make_float2(fmaf(Mi.m0, rf, Mi.m1 * rf1), fmaf(Mi.m2, rf, Mi.m3 * rf1));
        }
    }
}

// 5 CTAs per SM (at most 51 registers)
template <bool RG>
__global__ void __launch_bounds__(kMpThreads, 5)
mp_residual_kernel(MpArgs p)
{
    __shared__ double sx[kMpTile + 4];
    pdl_wait();
    pdl_release();                                // one wave of persistent CTAs: the successor may queue now
    // (resolved into locals: the argument block itself stays read-only)
    const int s = p.ctr ? *p.ctr : p.sweep;
    const XView xv = x_view(s, p.max_sweeps, p.X0f, p.xout, p.oss, p.ors, p.rg);
    if (__ldg(p.live + s + 1) == 0) return;       // every system has finished
    const bool fused0 = p.first_fused && s == 0;  // the fused sweep 0 formed r_0 of the systems it solved
    if (fused0 && __ldg(p.nfail) == 0) return;
    const int64_t tiles = (p.n + kMpTile - 1) / kMpTile;
    for (int64_t blk = blockIdx.x; blk < p.m * tiles; blk += gridDim.x) {
        const int64_t j = blk / tiles;
        if (__ldg(p.fin + j) != 0) continue;
        if (fused0 && !__ldg(p.fail + j)) continue;
        residual_tile<RG>(p, s, xv, j, blk - j * tiles, sx);
        __syncthreads();
    }
}

// End of a graph-driven sweep: advance the counter and tell the enclosing
// while node whether another sweep runs (a sweep remains and a system is
// still running).
__global__ void mp_advance_kernel(MpArgs p, cudaGraphConditionalHandle h)
{
    pdl_wait();
    const int s = *p.ctr + 1;
    *p.ctr = s;
    cudaGraphSetConditional(h, (s < p.max_sweeps && p.live[s] > 0) ? 1u : 0u);
}

// r = y - A x (FP64 FMA chain; a null outer band is zero).  Bands and y use the caller's layout (ss, rs);
// x and r use (xss, xrs).
__global__ void __launch_bounds__(kMpThreads)
residual_kernel(const double* __restrict__ a, const double* __restrict__ b, const double* __restrict__ c,
                const double* __restrict__ d, const double* __restrict__ e, const double* __restrict__ y,
                const double* __restrict__ x, double* __restrict__ r, int64_t m, int64_t n, int64_t ss, int64_t rs,
                int64_t xss, int64_t xrs)
{
    const int64_t total = m * n;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
         q += (int64_t)gridDim.x * blockDim.x) {
        int64_t j, i;
        if (rs == 1) { j = q / n; i = q - j * n; } else { i = q / m; j = q - i * m; }
        const int64_t g = j * ss + i * rs;
        const int64_t gx = j * xss + i * xrs;
        double v = y[g];
        v = fma(-c[g], x[gx], v);
        if (a && i >= 2) v = fma(-a[g], x[gx - 2 * xrs], v);
        if (i >= 1) v = fma(-b[g], x[gx - xrs], v);
        if (i + 1 < n) v = fma(-d[g], x[gx + xrs], v);
        if (e && i + 2 < n) v = fma(-e[g], x[gx + 2 * xrs], v);
        r[gx] = v;
    }
}

// Report of a solve: one pass over a tile of rows of system j forms
// r = y - A x (the FMA order of residual_kernel), the per-system maxima of
// |r_i|, sum_k |A_ik| and |x_i| (float bit patterns), and moves x to y.  Only
// the tile's own rows of y are written, after they were read.  Rounding to
// float is monotone, so the maxima are taken on the doubles' bits (no FP64
// compare or conversion per row; nans do not count, as with fmaxf) and
// converted once per warp.  Bound by its FP64 work, 5 FMA per row: the row
// sums, 4 more, are formed in FP64 only for the rows whose single-precision
// estimate can be the warp's largest.  Replaces a residual, a norm and a copy
// kernel that read the bands twice and passed r through memory (m=100
// n=30001: 48 us, 80 % of the FP64 pipe; 91 us with every row sum in FP64 and
// its loads behind branches; the three kernels ~130 us).
__device__ __forceinline__ void fold_max(unsigned long long& m, double v)
{
    const unsigned long long b = absbits(v);
    if (b <= 0x7FF0000000000000ull) m = max(m, b);
}

// |v| truncated to float (0 below 2^-126, inf from 2^128 on and for nans)
__device__ __forceinline__ float abs_estimate(double v)
{
    const unsigned h = (unsigned)__double2hiint(v) & 0x7FFFFFFFu;
    const unsigned f = ((h - (896u << 20)) << 3) | ((unsigned)__double2loint(v) >> 29);
    return h < (897u << 20) ? 0.0f : __uint_as_float(h >= (1151u << 20) ? 0x7F800000u : f);
}

constexpr int kReportRows = 4;                    // rows per thread

__global__ void __launch_bounds__(kMpThreads)
report_kernel(const double* __restrict__ a, const double* __restrict__ b, const double* __restrict__ c,
              const double* __restrict__ d, const double* __restrict__ e, const double* __restrict__ X, double* y,
              int64_t m, int64_t n, int64_t ss, int64_t rs, unsigned* __restrict__ rn, unsigned* __restrict__ an,
              unsigned* __restrict__ xn)
{
    constexpr int kTile = kReportRows * kMpThreads;
    const int64_t tiles = (n + kTile - 1) / kTile;
    for (int64_t blk = blockIdx.x; blk < m * tiles; blk += gridDim.x) {
        const int64_t j = blk / tiles, i0 = (blk - j * tiles) * kTile + threadIdx.x;
        const double* __restrict__ x = X + j * n;
        unsigned long long rm = 0ull, am = 0ull, xm = 0ull;
        float est[kReportRows];
        // every load of a row first (slots outside the system are zeros)
#pragma unroll 2
        for (int u = 0; u < kReportRows; u++) {
            const int64_t i = i0 + u * kMpThreads, g = j * ss + i * rs;
            est[u] = 0.0f;
            if (i < n) {
                const bool l2 = i >= 2, l1 = i >= 1, r1 = i + 1 < n, r2 = i + 2 < n;
                const double wc = c[g], yv = y[g], xv = x[i];
                const double wa = a && l2 ? a[g] : 0.0, wb = l1 ? b[g] : 0.0;
                const double wd = r1 ? d[g] : 0.0, we = e && r2 ? e[g] : 0.0;
                const double xa = a && l2 ? x[i - 2] : 0.0, xb = l1 ? x[i - 1] : 0.0;
                const double xd = r1 ? x[i + 1] : 0.0, xe = e && r2 ? x[i + 2] : 0.0;
                double v = fma(-wc, xv, yv);
                v = fma(-wa, xa, v);
                v = fma(-wb, xb, v);
                v = fma(-wd, xd, v);
                v = fma(-we, xe, v);
                est[u] = (abs_estimate(wc) + abs_estimate(wa)) + (abs_estimate(wb) + abs_estimate(wd)) +
                         abs_estimate(we);
                fold_max(rm, v); fold_max(xm, xv);
                y[g] = xv;
            }
        }
        // (an estimate is within 2^-20 of its sum unless terms were below
        // 2^-126 or above 2^128: then every row counts)
        float top = est[0];
#pragma unroll
        for (int u = 1; u < kReportRows; u++) top = fmaxf(top, est[u]);
        top = warp_max(top);
        const float least = top > 1e-30f && top < FLT_MAX ? top * (1.0f - 0x1p-19f) : -1.0f;
#pragma unroll
        for (int u = 0; u < kReportRows; u++) {
            const int64_t i = i0 + u * kMpThreads, g = j * ss + i * rs;
            if (i < n && est[u] >= least) {
                double rowsum = fabs(c[g]);
                if (a && i >= 2) rowsum += fabs(a[g]);
                if (i >= 1) rowsum += fabs(b[g]);
                if (i + 1 < n) rowsum += fabs(d[g]);
                if (e && i + 2 < n) rowsum += fabs(e[g]);
                fold_max(am, rowsum);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            rm = max(rm, __shfl_xor_sync(0xffffffffu, rm, o));
            am = max(am, __shfl_xor_sync(0xffffffffu, am, o));
            xm = max(xm, __shfl_xor_sync(0xffffffffu, xm, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomic_max_pos(&rn[j], (float)__longlong_as_double((long long)rm));
            atomic_max_pos(&an[j], (float)__longlong_as_double((long long)am));
            atomic_max_pos(&xn[j], (float)__longlong_as_double((long long)xm));
        }
    }
}

// The batch's report from the per-system values (one CTA)
__global__ void __launch_bounds__(kMpThreads)
summary_kernel(MpArgs p, const unsigned* __restrict__ rn, MpSummary* out)
{
    __shared__ MpSummary part[kMpThreads / 32];
    MpSummary s{0, 1, 0.0f, 0, 0.0};
    auto fold = [&](int sweeps, int converged, float est, double resid) {
        s.sweeps = max(s.sweeps, sweeps);
        s.converged &= converged;
        s.est = est > s.est ? est : s.est;
        s.resid = resid > s.resid ? resid : s.resid;
    };
    for (int64_t j = threadIdx.x; j < p.m; j += kMpThreads) {
        const float rj = __uint_as_float(rn[j]), aj = __uint_as_float(rn[p.m + j]), xj = __uint_as_float(rn[2 * p.m + j]);
        const double den = (double)aj * (double)xj;
        fold(p.fin[j], p.status[j] == 1, p.est[j], den > 0.0 ? rj / den : (rj > 0.0f ? 1.0 : 0.0));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        fold(__shfl_xor_sync(0xffffffffu, s.sweeps, o), __shfl_xor_sync(0xffffffffu, s.converged, o),
             __shfl_xor_sync(0xffffffffu, s.est, o), __shfl_xor_sync(0xffffffffu, s.resid, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kMpThreads / 32; k++) fold(part[k].sweeps, part[k].converged, part[k].est, part[k].resid);
        s.gave_up = p.err ? *p.err : 0;
        *out = s;
    }
}

// shared memory of the pass kernel: L, U (float4) and Y (float2) per block row
size_t mp_pass_smem(int rows) { return (size_t)mp_pass_rows(rows) * (2 * sizeof(float4) + sizeof(float2)); }

template <int RPT>
cudaError_t launch_mp_pass_rpt(const MpPassArgs& p, int threads, int64_t blocks, cudaStream_t s)
{
    const size_t smem = mp_pass_smem(p.TRmax);
    cudaError_t e = cudaFuncSetAttribute(mp_pass_kernel<RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)mp_pass_smem(kMpMaxRows));
    if (e != cudaSuccess) return e;
    blocks = std::min<int64_t>(blocks, mp_grid_cap((const void*)mp_pass_kernel<RPT>, threads, smem));
    e = launch_dependent(mp_pass_kernel<RPT>, (unsigned)blocks, threads, smem, s, p);
    count_launch();
    return e;
}

}  // namespace

cudaError_t launch_mp_init(const MpArgs& p, cudaStream_t s)
{
    const cudaError_t e = launch_dependent(mp_init_kernel, 152u * 2, kMpThreads, 0, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_first(const MpArgs& p, const MpWindows& g, cudaStream_t s)
{
    if (g.TRmax > kMpMaxRows) return cudaErrorInvalidValue;
    const int64_t items = p.m * g.nwin;
    if (items <= 0) return cudaSuccess;
    const size_t smem = mp_pass_smem(g.TRmax);
    auto kern = p.rg ? mp_first_kernel<true> : mp_first_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)mp_pass_smem(kMpMaxRows));
    if (e != cudaSuccess) return e;
    const int64_t blocks = std::min<int64_t>(items, mp_grid_cap((const void*)kern, kMpTryThreads, smem));
    e = launch_dependent(kern, (unsigned)blocks, kMpTryThreads, smem, s, p, g);
    count_launch();
    return e;
}

cudaError_t launch_mp_prep(const MpArgs& p, cudaStream_t s)
{
    const int64_t nb = (p.n + 1) / 2;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((p.m * nb + kMpThreads - 1) / kMpThreads, 152 * 16));
    const cudaError_t e = launch_dependent(p.rg ? mp_prep_kernel<true> : mp_prep_kernel<false>, (unsigned)blocks,
                                           kMpThreads, 0, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_rhs(const MpArgs& p, cudaGraphConditionalHandle windows, cudaGraphConditionalHandle full, bool gate,
                          cudaStream_t s)
{
    auto kern = p.rg ? mp_rhs_kernel<true> : mp_rhs_kernel<false>;
    const int64_t need = (p.m * ((p.n + 1) / 2) + kMpThreads - 1) / kMpThreads;
    const int64_t blocks = std::min<int64_t>(need, mp_grid_cap((const void*)kern, kMpThreads, 0));
    const cudaError_t e = launch_dependent(kern, (unsigned)blocks, kMpThreads, 0, s, p, windows, full, gate);
    count_launch();
    return e;
}

cudaError_t launch_mp_pass(const MpPassArgs& p, cudaStream_t s)
{
    if (p.TRmax > kMpMaxRows) return cudaErrorInvalidValue;
    int threads = kMpThreads;
    if (p.TRmax < threads) threads = std::max(32, (p.TRmax + 31) / 32 * 32);
    const int rpt = (p.TRmax + threads - 1) / threads;
    const int64_t items = p.m * p.G * p.nwin;
    if (items <= 0) return cudaSuccess;
    const int64_t blocks = items;
    if (rpt <= 1) return launch_mp_pass_rpt<1>(p, threads, blocks, s);
    if (rpt <= 2) return launch_mp_pass_rpt<2>(p, threads, blocks, s);
    if (rpt <= 4) return launch_mp_pass_rpt<4>(p, threads, blocks, s);
    if (rpt <= 8) return launch_mp_pass_rpt<8>(p, threads, blocks, s);
    return cudaErrorInvalidValue;
}

cudaError_t launch_mp_try(const MpPassArgs& p, cudaStream_t s)
{
    if (p.TRmax > kMpMaxRows) return cudaErrorInvalidValue;
    const int64_t items = p.m * p.nwin;
    if (items <= 0) return cudaSuccess;
    const size_t smem = mp_pass_smem(p.TRmax);
    cudaError_t e = cudaFuncSetAttribute(mp_try_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)mp_pass_smem(kMpMaxRows));
    if (e != cudaSuccess) return e;
    const int64_t blocks = std::min<int64_t>(items, mp_grid_cap((const void*)mp_try_kernel, kMpTryThreads, smem));
    // Uniform batches of at most two tiles per SM take the largest shared
    // memory of the SM.  Without that the general passes of a graph's sweeps are
    // up to a fifth slower in such batches (this kernel's 60 registers allow
    // four tiles, whose shared memory leaves the SM a smaller one; at the 48
    // registers of before it took the largest by itself), with it slower in
    // larger ones.  Coupled systems, us, with / without: 8 of 30000 rows 246 /
    // 279, 16 of 20000 262 / 296, 30 of 9000 235 / 269, 16 of 30000 (272 tiles)
    // 292 / 329; 20 of 30000 (340) 370 / 352, 64 of 30000 740 / 707; classes of a
    // ragged batch, several at once, 2203 / 2157.
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 0;
    const bool spare = !p.rg && items <= 2 * (int64_t)sms;
    e = launch_dependent_as(spare, mp_try_kernel, (unsigned)blocks, kMpTryThreads, smem, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_small(const MpArgs& p, cudaStream_t s)
{
    const int64_t nb = (p.n + 1) / 2;
    if (nb > kMpMaxRows) return cudaErrorInvalidValue;
    if (p.m <= 0) return cudaSuccess;
    const size_t smem = mp_pass_smem((int)nb);
    // short systems wait for a level's factors longer than they take to reduce
    // it (us, reduced again / replayed: 29583 ADI systems of 139 rows 297 / 310,
    // 40000 of 64 rows 143 / 146, 1024 of 512 rows 36.2 / 35.7, 4000 of 1000
    // rows 242 / 231, 4096 of 4096 rows 910 / 874)
    const bool keep = nb > kMpNarrow;
    auto kern = p.rg ? (keep ? mp_small_kernel<true, true> : mp_small_kernel<true, false>)
                     : (keep ? mp_small_kernel<false, true> : mp_small_kernel<false, false>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)mp_pass_smem(kMpMaxRows));
    if (e != cudaSuccess) return e;
    // large tiles hold two CTAs per SM (shared memory): twice the threads per
    // CTA keep as many warps resident as four CTAs of small tiles; tiles of at
    // most kMpNarrow block rows get 128 threads, so that more systems run at
    // once while each waits for its barriers (m=1024 n=512, interleaved: 8
    // instead of 4 CTAs per SM, one wave instead of two, 45.2 -> 38.3 us; at
    // n=2000 256 threads 154 us, 128 210); systems of fewer than 128 block
    // rows one thread per block row (whole warps)
    const int threads = nb >= 1024 ? kMpSmallThreadsMax : nb > kMpNarrow ? kMpThreads
                        : (int)std::min<int64_t>(128, std::max<int64_t>(32, (nb + 31) / 32 * 32));
    const int64_t blocks = std::min<int64_t>(p.m, mp_grid_cap((const void*)kern, threads, smem));
    e = launch_dependent(kern, (unsigned)blocks, threads, smem, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_xupdate(const MpArgs& p, cudaStream_t s)
{
    const int64_t tiles = (p.n + 4 * kMpThreads - 1) / (4 * kMpThreads);
    const int64_t blocks = std::min<int64_t>(p.m * tiles, mp_grid_cap((const void*)mp_xupdate_kernel, kMpThreads, 0));
    const cudaError_t e = launch_dependent(mp_xupdate_kernel, (unsigned)blocks, kMpThreads, 0, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_decide(const MpArgs& p, cudaStream_t s)
{
    const int64_t blocks = (p.m + kMpThreads - 1) / kMpThreads;
    const cudaError_t e = launch_dependent(mp_decide_kernel, (unsigned)blocks, kMpThreads, 0, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_residual(const MpArgs& p, cudaStream_t s)
{
    // one wave of CTAs striding over the tiles: a sweep after which every
    // system has finished returns at once through the live count
    const int64_t tiles = (p.n + kMpTile - 1) / kMpTile;
    auto kern = p.rg ? mp_residual_kernel<true> : mp_residual_kernel<false>;
    const int64_t blocks = std::min<int64_t>(p.m * tiles, mp_grid_cap((const void*)kern, kMpThreads, 0));
    const cudaError_t e = launch_dependent(kern, (unsigned)blocks, kMpThreads, 0, s, p);
    count_launch();
    return e;
}

cudaError_t launch_mp_advance(const MpArgs& p, cudaGraphConditionalHandle h, cudaStream_t s)
{
    const cudaError_t e = launch_dependent(mp_advance_kernel, 1u, 1u, 0, s, p, h);
    count_launch();
    return e;
}

cudaError_t launch_residual(const double* a, const double* b, const double* c, const double* d, const double* e,
                            const double* y, const double* x, double* r, int64_t m, int64_t n, int64_t ss,
                            int64_t rs, int64_t xss, int64_t xrs, cudaStream_t s)
{
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((m * n + kMpThreads - 1) / kMpThreads, 152 * 16));
    residual_kernel<<<(unsigned)blocks, kMpThreads, 0, s>>>(a, b, c, d, e, y, x, r, m, n, ss, rs, xss, xrs);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_report(const MpArgs& p, const double* X, unsigned* norms, MpSummary* out, cudaStream_t s)
{
    const int64_t tiles = (p.n + kReportRows * kMpThreads - 1) / (kReportRows * kMpThreads);
    const int64_t blocks = std::min<int64_t>(p.m * tiles, mp_grid_cap((const void*)report_kernel, kMpThreads, 0));
    report_kernel<<<(unsigned)blocks, kMpThreads, 0, s>>>(p.a, p.b, p.c, p.d, p.e, X, p.y, p.m, p.n, p.ss, p.rs, norms,
                                                          norms + p.m, norms + 2 * p.m);
    count_launch();
    summary_kernel<<<1, kMpThreads, 0, s>>>(p, norms, out);
    count_launch();
    return cudaGetLastError();
}

}  // namespace pcrp
