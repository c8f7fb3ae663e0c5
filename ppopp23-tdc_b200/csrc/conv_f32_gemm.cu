// Instances of conv_f32_gemm_kernel, the choice between them, and the launch.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <set>
#include <utility>
#include "conv_f32_gemm.h"
#include "conv_f32_gemm.cuh"
#include "errors.h"

namespace tdc {

namespace {

struct Form { int bm, bn; const void* fn[4]; };      // 1x1 (16-byte copies), 1x1, 3x3, any
#define TDC_FORM(BM_, BN_, TM_, TN_) {BM_, BN_, {(const void*)&conv_f32_gemm_kernel<BM_, BN_, TM_, TN_, 1, true>, (const void*)&conv_f32_gemm_kernel<BM_, BN_, TM_, TN_, 1, false>, \
                                                 (const void*)&conv_f32_gemm_kernel<BM_, BN_, TM_, TN_, 9, false>, (const void*)&conv_f32_gemm_kernel<BM_, BN_, TM_, TN_, 0, false>}}
const Form k_forms[] = {TDC_FORM(64, 128, 8, 8), TDC_FORM(32, 128, 4, 8), TDC_FORM(64, 64, 8, 4), TDC_FORM(32, 64, 4, 4)};

std::mutex g_mu;
std::set<std::pair<int, const void*>> g_opted;

size_t smem_of(const Form& f, bool three, int kc) {
    const int bk = three ? 36 : 32;
    return sizeof(float) * ((size_t)GEMM_STAGES * bk * (f.bm + GEMM_WPAD + f.bn) + (kc > 1 ? (size_t)f.bm * f.bn : 0));
}

}  // namespace

bool gemm_fits(const Shape& s) {
    return s.R <= 7 && s.S <= 7 && (long long)s.B * s.Ho() * s.Wo() < (1ll << 30) && (long long)s.C * s.R * s.S < (1ll << 24) &&
           (long long)s.H * s.W < (1ll << 30);
}

// Estimate of a launch's time in SM clocks: waves of tiles over the SMs, a wave being rows x (the slower of FMAs at 128 per
// clock and of shared loads at four clocks per warp and 16-byte load, plus the input copies), but no less than the chain of
// stages of a lone CTA.  Clusters of eight do not find room on every SM.  Constants fitted to 185 layers of batch 1 - 64,
// 7 - 112 pixels and 16 - 2048 channels timed in every form (3,000 timings): the form picked is 3 % slower than the fastest
// on average.
static double gemm_clocks(const Shape& s, const GemmTile& t) {
    const bool three = s.R == 3 && s.S == 3, one = s.R == 1 && s.S == 1, vec = one && s.stride == 1 && (s.H * s.W) % 4 == 0;
    const int tm = t.bm == 64 ? 8 : 4, tn = t.bn == 128 ? 8 : 4, bk = three ? 36 : 32;
    const double rows = (double)s.C * s.R * s.S, npos = (double)s.B * s.Ho() * s.Wo();
    const double per = std::ceil(std::ceil(rows / bk) / t.kc) * bk;
    const double ctas = std::ceil(npos / t.bn) * std::ceil((double)s.K / t.bm) * t.kc;
    const size_t smem = sizeof(float) * ((size_t)GEMM_STAGES * bk * (t.bm + GEMM_WPAD + t.bn) + (t.kc > 1 ? (size_t)t.bm * t.bn : 0));
    const double per_sm = std::min(2.0, std::floor(227.0 * 1024 / (double)(smem + 1024)));
    const double sms = t.kc == 1 ? 148.0 : (t.kc == 2 ? 146.0 : (t.kc == 4 ? 136.0 : 128.0));
    const double row = 1.14 * std::max(t.bm * (double)t.bn / 128.0, 4.0 * (tm / 4 + tn / 4) * 4.0) + t.bn / 32.0 * (vec ? 0.15 : (one ? 1.2 : 1.0));
    const double chain = t.bm == 64 && t.bn == 128 ? 190.0 : (t.bm + t.bn == 96 ? 17.0 : 60.0);
    const double waves = std::ceil(ctas / (sms * per_sm)), last = std::ceil((ctas - (waves - 1.0) * sms * per_sm) / sms);
    return 2700.0 + per * ((waves - 1.0) * std::max(per_sm * row, chain) + std::max(last * row, chain)) +
           (t.kc == 1 ? 0.0 : (t.kc == 2 ? 1730.0 : 2350.0)) + waves * 1000.0;
}

GemmTile gemm_choose(const Shape& s) {
    GemmTile best{};
    double least = 0.0;
    for (const Form& f : k_forms)
        for (int kc = 1; kc <= 8; kc *= 2) {
            if (kc > 1 && s.C * s.R * s.S < 32 * kc) break;           // a rank without a stage
            const GemmTile t{f.bm, f.bn, kc};
            const double c = gemm_clocks(s, t);
            if (!best.bm || c < least) { best = t; least = c; }
        }
    return best;
}

// Measured against conv_f32_kernel on its table's (or model's) tile on 214 layers: 1.1 - 6 times as fast on all but 13.
// Those have filters beyond 3x3, whose windows the rectangles of conv_f32_kernel read once where this kernel gathers every
// row (with torch's filter layout this kernel wins all the same), or one tile of 64 channels that their outputs fill to five
// eighths at most (33 - 40 channels, above 4 GFLOP): the rectangles of conv_f32_kernel go in steps of 4 channels.
bool gemm_wins(const Shape& s, bool channel_last) {
    if (!gemm_fits(s)) return false;
    if (s.R * s.S > 9) return !channel_last || s.C < 16;
    const bool half_empty = s.K > 32 && s.K <= 64 * 5 / 8;
    return !(s.R == 3 && half_empty && 18.0 * s.C * s.K * s.B * s.Ho() * s.Wo() > 4e9);
}

int gemm_launch(const ConvArgs& base, const Shape& s, const GemmTile& t, int device, cudaStream_t stream) {
    const Form* f = nullptr;
    for (const Form& q : k_forms) if (q.bm == t.bm && q.bn == t.bn) f = &q;
    if (!f || (t.kc != 1 && t.kc != 2 && t.kc != 4 && t.kc != 8)) return fail(TDC_ERR_TILE, "no tile of %d channels x %d positions over %d CTAs is built", t.bm, t.bn, t.kc);
    if (!gemm_fits(s)) return fail(TDC_ERR_UNSUPPORTED, "shape too large for this kernel");
    GemmArgs g{};
    g.c = base;
    const bool three = s.R == 3 && s.S == 3;
    const int bk = three ? 36 : 32;
    g.rows = s.C * s.R * s.S;
    g.kc = t.kc;
    const int stages = (g.rows + bk - 1) / bk;
    g.rows_per_rank = (stages + t.kc - 1) / t.kc * bk;
    g.n_chb = (s.K + t.bm - 1) / t.bm;
    g.npos = (uint32_t)((long long)s.B * s.Ho() * s.Wo());
    g.stride = s.stride;
    g.fd_img = tdc_tc::fastdiv_make((uint32_t)(s.Ho() * s.Wo()));
    g.fd_wo = tdc_tc::fastdiv_make((uint32_t)s.Wo());
    g.fd_rs = tdc_tc::fastdiv_make((uint32_t)(s.R * s.S));
    g.fd_s = tdc_tc::fastdiv_make((uint32_t)s.S);
    g.fd_chb = tdc_tc::fastdiv_make((uint32_t)g.n_chb);
    g.out_vec = (s.Ho() * s.Wo()) % 4 == 0 && base.y_vec && (!base.residual || reinterpret_cast<uintptr_t>(base.residual) % 16 == 0);
    const bool vec = s.R == 1 && s.S == 1 && s.stride == 1 && s.pad == 0 && (s.H * s.W) % 4 == 0 && reinterpret_cast<uintptr_t>(base.x) % 16 == 0;
    const void* fn = f->fn[s.R == 1 && s.S == 1 ? (vec ? 0 : 1) : (three ? 2 : 3)];
    const long long ctas = (long long)((g.npos + t.bn - 1) / t.bn) * g.n_chb * t.kc;
    if (ctas >= (1ll << 31)) return fail(TDC_ERR_TILE, "grid too large");
    const size_t smem = smem_of(*f, three, t.kc);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_opted.insert({device, fn}).second) {
            const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_of(k_forms[0], true, 2));
            if (e != cudaSuccess) return fail(TDC_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        }
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ctas); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = t.kc; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = t.kc > 1 ? 2 : 1;
    void* args[] = {&g};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    return e == cudaSuccess ? TDC_OK : fail(TDC_ERR_CUDA, "launch: %s", cudaGetErrorString(e));
}

}  // namespace tdc
