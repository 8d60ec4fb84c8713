// lbm_variants.cuh -- the compiled step-kernel variants and how to launch them.
//
// Each translation unit variants_*.cu instantiates one group of variants of
// lbm::step_kernel (lattice x storage format) and exposes a pick_* function
// that returns the launcher for a requested tiling; splitting them keeps the
// build parallel.  lbm_capi.cu only sees the Launcher records.
#pragma once

#include <cstddef>

namespace lbm {

struct Launcher {
    void *fn = nullptr;      // plain step
    void *fn_mon = nullptr;  // step that also accumulates the per-step monitor sums
    size_t smem = 0;
    int tx = 0, ty = 0, stages = 0, pop_buffers = 2;
};

// Every compiled kernel variant: (lattice, tile x, tile y, TMA stages,
// population-plane code, storage).  Population-plane code 1 = one plane,
// 3 CTAs/SM; 2 = two planes, 2 CTAs/SM; 4 = one plane, 4 CTAs/SM.  Storage
// codes: 0 FP32, 1 FP16, 2 BF16.
struct Variant {
    int Q, tx, ty, stages, npb, storage;
};
constexpr Variant kVariants[] = {
    {19, 32, 8, 2, 1, 0}, {19, 32, 8, 3, 1, 0}, {19, 32, 8, 3, 2, 0}, {19, 32, 8, 2, 2, 0}, {19, 32, 8, 2, 4, 0},
    {19, 16, 8, 2, 1, 0}, {19, 8, 8, 2, 1, 0},  {27, 32, 8, 2, 1, 0}, {27, 32, 8, 2, 2, 0}, {27, 16, 8, 2, 1, 0},
    {27, 8, 8, 2, 1, 0},  {19, 32, 8, 2, 1, 1}, {19, 32, 8, 3, 1, 1}, {19, 16, 8, 2, 1, 1}, {27, 32, 8, 2, 1, 1},
    {27, 16, 8, 2, 1, 1}, {19, 32, 8, 2, 1, 2}, {19, 32, 8, 3, 1, 2}, {19, 16, 8, 2, 1, 2}, {27, 32, 8, 2, 1, 2},
    {27, 16, 8, 2, 1, 2}, {19, 32, 8, 2, 4, 1}, {19, 32, 8, 2, 4, 2}};

// fo: the handle's function-object bits (LBM_FO_*).
bool pick_q19_f32(int tx, int ty, int stages, int npb, unsigned fo, int mean_bits, Launcher &out);
bool pick_q27_f32(int tx, int ty, int stages, int npb, unsigned fo, int mean_bits, Launcher &out);
bool pick_f16(int Q, int tx, int ty, int stages, int npb, unsigned fo, int mean_bits, Launcher &out);
bool pick_bf16(int Q, int tx, int ty, int stages, int npb, unsigned fo, int mean_bits, Launcher &out);

#ifdef __CUDACC__
template <int Q, int TX, int TY, int NS, int FO, typename MeanT, bool MON, int NPB, int MINB, typename ST>
void *kernel_fn()
{
    return reinterpret_cast<void *>(&step_kernel<Q, TX, TY, NS, FO, MeanT, MON, NPB, MINB, ST>);
}

// The function-object kernel for a set of function objects: none; exactly
// S, SMean, k and kMean (code 2: no run-time checks); any set with momentsMean
// (code 3); any other set (code 1).  Code 3 is apart because the old means of
// the moments take ten registers (FP64: twenty) that the other sets' kernels
// would spill for (D3Q19 256^3, k and kMean in FP64: 321 us per step alone,
// 393 with them).
constexpr unsigned kFoFour = 0x0Fu;  // LBM_FO_S | LBM_FO_SMEAN | LBM_FO_K | LBM_FO_KMEAN
constexpr unsigned kFoMomentsMean = 0x10u;  // LBM_FO_MOMENTSMEAN

template <int Q, int TX, int TY, int NS, int NPB, int MINB, typename ST, int FO>
void pick_means(Launcher &l, int mean_bits)
{
    if (mean_bits == 64) {
        // FP64 old means of all moments: with the six of SMean 20 registers
        // more are worth a CTA.  us per step of 32-wide tiles at 3 / 2 CTAs
        // per SM, best of the z-chunks 2 to 26, all five function objects:
        // D3Q27 64^3 17.2 / 16.3, 136x120x128 154.6 / 152.1, 256^3 1043 /
        // 1039, D3Q19 256^3 1049 / 1030, D3Q27 256^3 in FP16 storage 925 /
        // 944; at the default chunk of 256^3 2 CTAs take 0.94-0.96 of the
        // time.  Sets without SMean gain on small meshes and lose on large
        // ones (momentsMean alone, D3Q27: 64^3 14.3 / 13.1, 96^3 39.8 / 46.2,
        // 256^3 685 / 748, in FP16 storage 611 / 701).  16- and 8-wide tiles
        // run the same within 3%.
        constexpr int MB = FO == 3 && MINB > 2 ? 2 : MINB;
        l.fn = kernel_fn<Q, TX, TY, NS, FO, double, false, NPB, MB, ST>();
        l.fn_mon = kernel_fn<Q, TX, TY, NS, FO, double, true, NPB, MB, ST>();
    } else {
        l.fn = kernel_fn<Q, TX, TY, NS, FO, float, false, NPB, MINB, ST>();
        l.fn_mon = kernel_fn<Q, TX, TY, NS, FO, float, true, NPB, MINB, ST>();
    }
}

template <int Q, int TX, int TY, int NS, int NPB, int MINB, typename ST>
Launcher pick_fo(unsigned fo, int mean_bits)
{
    Launcher l;
    l.tx = TX;
    l.ty = TY;
    l.stages = NS;
    l.pop_buffers = NPB;
    l.smem = SmemLayout<Q, TX, TY, NS, NPB, ST>::bytes;
    if (!fo) {
        l.fn = kernel_fn<Q, TX, TY, NS, 0, float, false, NPB, MINB, ST>();
        l.fn_mon = kernel_fn<Q, TX, TY, NS, 0, float, true, NPB, MINB, ST>();
    } else if (fo == kFoFour) {
        pick_means<Q, TX, TY, NS, NPB, MINB, ST, 2>(l, mean_bits);
    } else if (fo & kFoMomentsMean) {
        pick_means<Q, TX, TY, NS, NPB, MINB, ST, 3>(l, mean_bits);
    } else {
        pick_means<Q, TX, TY, NS, NPB, MINB, ST, 1>(l, mean_bits);
    }
    return l;
}

#define LBM_VARIANT(QQ, TXX, TYY, NSS, NPBCODE, NPB, MINB, ST)                                  \
    if (Q == QQ && tx == TXX && ty == TYY && stages == NSS && npb == NPBCODE) {                 \
        out = pick_fo<QQ, TXX, TYY, NSS, NPB, MINB, ST>(fo, mean_bits);                          \
        out.pop_buffers = NPBCODE;                                                              \
        return true;                                                                            \
    }
#endif

}  // namespace lbm
