// pcr_f64.cu -- faithful FP64 PCR-Penta stride kernel for sm_103a.
//
// One kernel serves both reference paths:
//   * whole (sub)systems in shared memory, strides + final step, x written
//     (the reference's pcr_penta, kernel.cu:32-154, and its second stage
//     pcr_penta_splitting_2nd_stage, kernel.cu:665-791);
//   * windows with halos of a long system: K strides fused per global-memory
//     pass, state written to a scratch buffer (the reference's stage-1
//     splitting kernels, kernel.cu:158-659, which run one stride per tile
//     sweep and one CTA per system).
//
// After s strides the rows of a system that are congruent mod G = 2^s form
// independent subsystems (row i then couples i +- G, i +- 2G only), so every
// pass works on a subsystem: rows  base + r + t*G,  t = 0 .. n_r-1.  Stride
// tests such as "i - delta >= 0" are exact in local coordinates
// (t - delta' >= 0 with delta = G*delta'), so a pass at level G performs the
// same operations on the same values as the global stride would.
//
// Arithmetic.  Each stride forms the reference's Reductions I, II, III
// (kernel.cu:68-140) with every product, sum and IEEE quotient rounded on its
// own (no FMA contraction), in the reference's order of evaluation.  The two
// neighbour combinations a row needs, R1(i) (rows i-2d, i-d, i) and R2(i)
// (rows i, i+d, i+2d), are the same combination T(m) centred on m = i-d and
// m = i+d, built from identical expressions (compare kernel.cu:77-79 with
// kernel.cu:103-105), so T(m) is formed once per row in phase A and shared
// through shared memory in phase B: 4 quotients per row and stride instead of
// the reference's 6, with bit-identical results.
//
// What bounds it.  One FP64 warp instruction takes 62 cycles of an SM
// sub-partition on this part, and the stride's 36 products and sums and 4
// quotients (an FP64 division: 8.6 such slots) used to keep that pipe 87 %
// busy.  The integer pipe runs beside it, so the quotients and 18 of the 20
// products are formed there (ieee_int.cuh: correctly rounded, the same bits;
// one product 25 instructions, one quotient 40) and 16 sums and 2 products stay
// FP64.  A dense stride now issues ~1,200 warp instructions per 32 rows, with
// the FP64 pipe 67 % and the integer ALU 62 % busy (4 CTAs of 256 threads per
// SM; what is left is the latency of the row's dependent chains between two
// barriers).  Measured, before and after: m=64 n=2^20 weakly dominant 91.7 ->
// 33.9 ms, m=256 n=65536 19.8 -> 7.8 ms, m=1024 n=512 interleaved 0.535 -> 0.264
// ms; a dense two-stride pass at m=4 n=2^20 1.00 -> 0.37 ms.
//
// The reference's multiplier registers, which outlive a stride and are reused
// when a pivot is exactly zero (kernel.cu:122,129), are formed again when that
// happens (pcr_tile), not kept.
#include "pcr_tile.cuh"

namespace pcrp {
namespace {

// CTAs per SM the register budget is set for: as many as shared memory holds
// (100 bytes per row), at most 1024 threads.
template <int CAP, bool kFew, bool kTri, bool kWindow = false>
__global__ void __launch_bounds__(kMaxThreads, CAP > 1024 ? 1 : CAP > 544 ? 2 : 4)
pcr_pass_kernel(const PcrPassArgs p)
{
    extern __shared__ __align__(16) unsigned char pcr_smem[];
    const uint32_t blk = blockIdx.x, nwin = (uint32_t)p.nwin, item = blk / nwin, w = blk - item * nwin;
    const uint32_t j = item >> p.lg, r = item & ((1u << p.lg) - 1);
    pcr_tile<CAP, false, kFew, kTri, kWindow>(p, j, r, w, *reinterpret_cast<TileRows<CAP>*>(pcr_smem));
}

constexpr int kShortRows = 2048;          // rows of a short system

template <int CAP, bool kFew, bool kTri, bool kWindow = false>
cudaError_t launch_tiles(const PcrPassArgs& p, int threads, int64_t blocks, cudaStream_t s)
{
    // per-device attribute, for more than the default 48 KB; cheap, and legal
    // while a stream is being captured
    if (sizeof(TileRows<CAP>) > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(pcr_pass_kernel<CAP, kFew, kTri, kWindow>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)sizeof(TileRows<CAP>));
        if (e != cudaSuccess) return e;
    }
    pcr_pass_kernel<CAP, kFew, kTri, kWindow><<<(unsigned)blocks, threads, sizeof(TileRows<CAP>), s>>>(p);
    count_launch();
    return cudaGetLastError();
}

template <int CAP>
cudaError_t launch_cap(const PcrPassArgs& p, bool tridiagonal, int threads, int64_t blocks, cudaStream_t s)
{
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // One row case for all rows (zeros among the operands selected) for
    // launches of at most two warps per SM sub-partition, where a row's latency
    // counts and the FP64 pipe is not full (us, one case / per-case rows: 8
    // systems of 512 rows 58 / 81; 32 systems of 4096 rows, six warps,
    // 152 / 136), and for short pentadiagonal systems, many of whose rows are
    // near an end in the late strides and would each load another case's code
    // (4000 systems of 100 rows 157 / 316, 2000 of 512 464 / 511, 2000 of 1000
    // 968 / 1135, 500 of 2000 581 / 609, 300 of 4000 737 / 708).  Tridiagonal
    // batches have a kernel of their own: their rows issue little FP64 work (8
    // systems of 512 rows 71 us by one case for all, 41 by theirs).
    const bool few = blocks * (threads / 32) <= 8 * (int64_t)sms;
    const bool shorts = p.n <= kShortRows;
    if (tridiagonal) return launch_tiles<CAP, false, true>(p, threads, blocks, s);
    if (few || shorts) return launch_tiles<CAP, true, false>(p, threads, blocks, s);
    // window passes of the tuned plans' tiles (512 rows) have a kernel without the finish
    constexpr bool tuned = CAP == 544;
    if (tuned && !p.final_step) return launch_tiles<CAP, false, false, tuned>(p, threads, blocks, s);
    return launch_tiles<CAP, false, false>(p, threads, blocks, s);
}

}  // namespace

int pcr_max_smem_rows() { return 1920; }

cudaError_t launch_pcr_pass(const PcrPassArgs& p, int threads, cudaStream_t s, bool tridiagonal)
{
    if (threads <= 0 || threads > kMaxThreads) threads = kMaxThreads;
    threads = (threads + 31) / 32 * 32;
    if (p.TRmax < threads) threads = (p.TRmax + 31) / 32 * 32;   // small (sub)systems: no idle warps
    while ((p.TRmax + threads - 1) / threads > kMaxRowsPerThread && threads < kMaxThreads) threads += 32;
    // as many warps as the rows per thread need (376 rows: two rounds of 192
    // threads, not of 256)
    const int rounds = (p.TRmax + threads - 1) / threads;
    threads = ((p.TRmax + rounds - 1) / rounds + 31) / 32 * 32;
    if (p.TRmax > pcr_max_smem_rows()) return cudaErrorInvalidValue;
    const int64_t blocks = p.m * p.G * p.nwin;
    if (blocks <= 0) return cudaSuccess;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    if (p.TRmax <= 32) return launch_cap<32>(p, tridiagonal, threads, blocks, s);
    if (p.TRmax <= 64) return launch_cap<64>(p, tridiagonal, threads, blocks, s);
    if (p.TRmax <= 128) return launch_cap<128>(p, tridiagonal, threads, blocks, s);
    if (p.TRmax <= 256) return launch_cap<256>(p, tridiagonal, threads, blocks, s);
    if (p.TRmax <= 384) return launch_cap<384>(p, tridiagonal, threads, blocks, s);
    if (p.TRmax <= 544) return launch_cap<544>(p, tridiagonal, threads, blocks, s);
    if (p.TRmax <= 1024) return launch_cap<1024>(p, tridiagonal, threads, blocks, s);
    return launch_cap<1920>(p, tridiagonal, threads, blocks, s);
}

}  // namespace pcrp
