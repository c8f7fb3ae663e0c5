// Convolution kernels on packed activations (pk.h describes the format; conv_tc.cu the algorithm, the operand layout and the
// accumulators, which are the same here).
//
// conv_pk_kernel: one CTA per SM walks a list of tiles (MT x 128 positions x NT output channels).
//   warp 0        producer: one lane issues the bulk copies of a stage — four runs of positions (two groups of 8 channels x
//                 hi, lo) per channel block and the filter blocks — and never waits for anything but a free stage;
//   warps 1, 2    issue the MMAs of position tiles 0 and 1;
//   warp 3        owns tensor memory;
//   warps 4-19    drain it: scale, shift, residual, ReLU, the next layer's split, 16-byte stores.
// There are no loader warps: what paced the kernels of conv_tc.cu (85-90 % busy converting and indexing, one latency chain
// per channel block) is gone, and what is left is the slowest of the copies, the MMAs and the epilogue's stores.
#pragma once
#include "pk.h"

namespace tdc_pk {
using namespace tdc_tc;

constexpr int PK_WARPS = 20, PK_THREADS = 32 * PK_WARPS, PK_EW0 = 4, PK_GROUPS = 4, PK_EPI = 512;
constexpr int PK_HEADER = 1024;
constexpr int PK_MAXNS = 8;
constexpr int PK_MAXRES = 32;

__device__ __forceinline__ void pk_tile_of(const Args& a, int mt_cap, long long t, long long& g0, int& cnt, int& ocb) {
    long long tg = t;
    ocb = 0;
    if (a.n_ocb > 1) { tg = (long long)fastdiv((uint32_t)t, a.fd_nocb); ocb = (int)(t - tg * a.n_ocb); }
    if (tg < a.full_groups) { g0 = tg * (mt_cap * M_TILE); cnt = mt_cap; }
    else {
        const long long first = a.tail_first + (tg - a.full_groups) * a.tail_cnt, left = a.pt_total - first;
        g0 = first * M_TILE;
        cnt = left < a.tail_cnt ? (int)left : a.tail_cnt;
    }
}

// With pooling (POOL) a tile is 128 columns of an even row and of the row below it, its two position tiles one above the other.
template <int POOL> __device__ __forceinline__ void tile_at(const Args& a, int mt_cap, long long t, long long& g0, int& cnt, int& ocb, int& img, int& pair, int& seg) {
    if (!POOL) { img = pair = seg = 0; pk_tile_of(a, mt_cap, t, g0, cnt, ocb); return; }
    img = (int)fastdiv((uint32_t)t, a.fd_timg);
    pair = (int)t - img * a.t_img;
    seg = 0;
    if (a.nseg > 1) { const int r = pair; pair = r / a.nseg; seg = r - pair * a.nseg; }
    g0 = (long long)img * a.sp.Lp + 2ll * pair * a.sp.Wp + seg * M_TILE;
    cnt = 2; ocb = 0;
}
// The tiles of a CTA.  With pooling it walks down the images: `t` to `end`, of which those before `first` only bring along the
// row above (3x3 windows).
struct Walk { long long t, first, end, step; };
template <int POOL> __device__ __forceinline__ Walk walk_of(const Args& a) {
    if (!POOL) return Walk{(long long)blockIdx.x, 0, a.ntiles, (long long)gridDim.x};
    const long long lo = a.ntiles * blockIdx.x / gridDim.x, hi = a.ntiles * (blockIdx.x + 1) / gridDim.x;
    const bool above = POOL == POOL_3x3 && lo < hi && lo % a.t_img != 0;
    return Walk{above ? lo - 1 : lo, lo, hi, 1};
}

// Taps of a channel block and the bytes of its filter part.
template <int MODE> __device__ __forceinline__ int taps_of(int parity) {
    if (MODE == MODE_S2) return (1 + (parity >> 1)) * (1 + (parity & 1));
    return MODE;
}
// Bytes of filter in front of channel block `cb` of parity `p` (MODE_S2: the parities' taps add up to 1, 2, 2, 4).
template <int MODE, int NT> __device__ __forceinline__ long long filter_offset(const Args& a, int ocb, int p, int cb) {
    constexpr long long unit = 64ll * NT;
    if (MODE == MODE_S2) {
        const int before = p == 0 ? 0 : (p == 1 ? 1 : (p == 2 ? 3 : 5));
        return unit * ((long long)ocb * 9 * a.cbl + (long long)before * a.cbl + (long long)taps_of<MODE>(p) * cb);
    }
    return unit * MODE * ((long long)ocb * a.nkb + cb);
}
// Positions the patch of a tile starts ahead of it, and positions it holds beyond it.
template <int MODE> __device__ __forceinline__ int patch_shift(const Space& sp, int parity) {
    if (MODE == MODE_3x3) return sp.Wp + 1;
    if (MODE == MODE_ROW3) return sp.Wp;
    if (MODE == MODE_4x4) return 2 * sp.Wp + 2;
    if (MODE == MODE_S2) return (parity >> 1) * sp.Wp + (parity & 1);
    return 0;
}
template <int MODE> __device__ __forceinline__ int patch_halo(const Space& sp, int parity) {
    if (MODE == MODE_3x3) return 2 * (sp.Wp + 1);
    if (MODE == MODE_ROW3) return 2 * sp.Wp;
    if (MODE == MODE_4x4) return 3 * (sp.Wp + 1);
    if (MODE == MODE_S2) return (parity >> 1) * sp.Wp + (parity & 1);
    return 0;
}
// Patch row of tap `tap` for the tile's first position.
template <int MODE> __device__ __forceinline__ int tap_row(int tap, int Wp, int pcols) {
    if (MODE == MODE_3x3) return (tap / 3) * Wp + tap % 3;
    if (MODE == MODE_ROW3) return tap * Wp;
    if (MODE == MODE_4x4) return (tap / 4) * Wp + tap % 4;
    if (MODE == MODE_S2) return pcols == 2 ? (tap >> 1) * Wp + (tap & 1) : tap * Wp;
    return 0;
}

// The MMAs of one channel block of one position tile: main += hi*hi and small += hi*lo in one MMA of width 2 NT, small +=
// lo*hi in another; odd channel blocks feed a second main accumulator where the host asked for two (conv_tc.cu: issue_block).
template <int NT, int MODE>
__device__ __forceinline__ void pk_issue(const Args& a, uint32_t d, uint32_t a_base, uint32_t b_base, uint32_t row16, int parity, bool second, bool first) {
    const uint32_t a_lbo = (uint32_t)a.P * 16u, b_lbo = (uint32_t)(2 * NT) * 16u, sbo = 128u;
    const uint32_t idesc_n = make_idesc<true>(NT), idesc_2n = make_idesc<true>(2 * NT);
    const uint64_t a_hi0 = make_desc(a_base, a_lbo, sbo) + row16;
    const uint64_t a_lo0 = make_desc(a_base + (uint32_t)a.P * 32u, a_lbo, sbo) + row16;
    const uint64_t b0 = make_desc(b_base, b_lbo, sbo);
    const int Wp = a.sp.Wp;
    auto one = [&](int tap, uint32_t off) {
        const uint64_t b = b0 + (uint64_t)(tap * 4 * NT);
        if (second) {
            mma_tf32<true>(d + 2 * NT, a_hi0 + off, b, idesc_n, (first && tap == 0) ? 0u : 1u);
            mma_tf32<true>(d + NT, a_hi0 + off, b + (uint64_t)NT, idesc_n, 1u);
            mma_tf32<true>(d + NT, a_lo0 + off, b, idesc_n, 1u);
        } else {
            mma_tf32<true>(d, a_hi0 + off, b, idesc_2n, (first && tap == 0) ? 0u : 1u);
            mma_tf32<true>(d + NT, a_lo0 + off, b, idesc_n, 1u);
        }
    };
    if constexpr (MODE == MODE_S2) {
        const int taps = taps_of<MODE>(parity), pcols = 1 + (parity & 1);
        for (int tap = 0; tap < taps; ++tap) one(tap, (uint32_t)tap_row<MODE>(tap, Wp, pcols));
    } else {
#pragma unroll
        for (int tap = 0; tap < MODE; ++tap) one(tap, (uint32_t)tap_row<MODE>(tap, Wp, 0));
    }
}

// Largest of n partial maxima (as bit patterns), one share per thread.
__device__ __forceinline__ unsigned int slots_max(const float* slots, int n, int idx, int threads) {
    unsigned int m = 0;
    for (int i = idx; i < n; i += threads) m = max(m, __float_as_uint(__ldcg(slots + i)) & 0x7fffffffu);
    return m;
}

// Where a computed position goes.
struct Where { long long same, out; bool in, valid; };        // same: position in the computed space; out: position (or NCHW offset) of the stored value
__device__ __forceinline__ Where place(const Args& a, long long g) {
    Where w;
    w.same = g; w.out = g;
    w.in = g < a.sp.total;
    w.valid = false;
    if (!w.in) return w;
    const uint32_t img = fastdiv((uint32_t)g, a.sp.fd_Lp);
    const uint32_t rem = (uint32_t)g - img * (uint32_t)a.sp.Lp;
    const int yy = (int)fastdiv(rem, a.sp.fd_Wp), xx = (int)rem - yy * a.sp.Wp;
    int b = (int)img, fy = yy, fx = xx;
    bool v = yy < a.sp.H && xx < a.sp.W;
    if (a.sp.split_B) {
        const int p = b >= 2 * a.sp.split_B ? 2 : 0, px = b >= (p + 1) * a.sp.split_B ? 1 : 0;
        b -= (p + px) * a.sp.split_B;
        fy = 2 * yy + (p >> 1); fx = 2 * xx + px;
        v = v && fy < a.sp.Hf && fx < a.sp.Wf;
    }
    w.valid = v;
    if (a.nchw) w.out = (long long)b * a.K * a.sp.Hf * a.sp.Wf + (long long)fy * a.sp.Wf + fx;
    else if (a.map == MAP_SPACE) w.out = ((long long)b * a.dsp.Lp) + (long long)fy * a.dsp.Wp + fx;
    else if (a.map == MAP_SPLIT)
        w.out = (long long)((((fy & 1) * 2 + (fx & 1)) * a.dsp.split_B) + b) * a.dsp.Lp + (long long)(fy >> 1) * a.dsp.Wp + (fx >> 1);
    return w;
}

// Pairs of floats.  The epilogue is bound by instruction issue (16 warps share four schedulers), and one instruction on a pair
// replaces two.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_of(float lo, float hi) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ f2 f2_of(uint32_t lo, uint32_t hi) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r; }
__device__ __forceinline__ void f2_get(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
// max(m, |a|, |b|); a NaN wins
__device__ __forceinline__ float max3_abs(float m, float a, float b) {
    float r;
    asm("{\n\t.reg .f32 p, q;\n\tabs.f32 p, %1;\n\tabs.f32 q, %2;\n\tmax.NaN.f32 %0, p, q, %3;\n\t}" : "=f"(r) : "f"(a), "f"(b), "f"(m));
    return r;
}

// Eight values times the power of two s -> one hi and one lo word: hi = fp16(c), lo = fp16((c - hi) * 2^11), c = v * s.
// (2^11 c and 2^11 hi are exact, and so is their difference: the fma rounds nothing.)
__device__ __forceinline__ void split8(const f2* v, float s, uint4& hi, uint4& lo) {
    const f2 s1 = f2_of(s, s), s2 = f2_of(s * 2048.f, s * 2048.f), m2 = f2_of(-2048.f, -2048.f);
    uint32_t h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float c0, c1;
        f2_get(f2_mul(v[k], s1), c0, c1);
        const __half2 hh = __floats2half2_rn(c0, c1);
        const float2 hf = __half22float2(hh);
        f2_get(f2_fma(f2_of(hf.x, hf.y), m2, f2_mul(v[k], s2)), c0, c1);
        const __half2 ll = __floats2half2_rn(c0, c1);
        h[k] = *reinterpret_cast<const uint32_t*>(&hh);
        l[k] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// 2 W channels from k0 on of one position: the residual of them, and every output asked for.  `ymax`: the largest magnitude of
// the values that are real.
template <int W>
__device__ __forceinline__ void residual(const Args& a, long long pos, bool valid, int k0, f2 (&rv)[W]) {
    const float* rp = a.res + (long long)(k0 >> 2) * a.res_plane + pos * 4;
#pragma unroll
    for (int q = 0; q < W / 2; ++q) {
        ulonglong2 t = make_ulonglong2(0ull, 0ull);
        if (valid && k0 + 4 * q < a.K) t = *reinterpret_cast<const ulonglong2*>(rp + (long long)q * a.res_plane);
        rv[2 * q] = t.x; rv[2 * q + 1] = t.y;
    }
}
template <int W>
__device__ __forceinline__ void store(const Args& a, const Where& w, int k0, f2 (&v)[W], float ys, float& ymax) {
    if (a.relu) {
#pragma unroll
        for (int k = 0; k < W; ++k) {
            float p, q;
            f2_get(v[k], p, q);
            v[k] = f2_of(max_nan(p, 0.f), max_nan(q, 0.f));
        }
    }
    float m = ymax;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        float p, q;
        f2_get(v[k], p, q);
        m = max3_abs(m, p, q);
    }
    if (w.valid) ymax = m;
    if (a.y && (w.valid || (a.map == MAP_SAME && w.in))) {
        char* p = a.y + (long long)(k0 >> 3) * 2 * a.y_plane + w.out * 16;
#pragma unroll
        for (int q = 0; q < W / 4; ++q) {
            uint4 hi, lo;
            split8(v + 4 * q, ys, hi, lo);
            if (!w.valid) hi = lo = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(p + (2 * q) * a.y_plane) = hi;
            *reinterpret_cast<uint4*>(p + (2 * q + 1) * a.y_plane) = lo;
        }
    }
    if (a.yf && w.valid) {
        float* p = a.yf + (long long)(k0 >> 2) * a.yf_plane + w.out * 4;
#pragma unroll
        for (int q = 0; q < W / 2; ++q)
            if (k0 + 4 * q < a.K) *reinterpret_cast<ulonglong2*>(p + (long long)q * a.yf_plane) = make_ulonglong2(v[2 * q], v[2 * q + 1]);
    }
    if (a.nchw && w.valid) {
        const long long HW = (long long)a.sp.Hf * a.sp.Wf;
        float* p = a.nchw + w.out + (long long)k0 * HW;
        const int n = a.K - k0;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            float lo, hi;
            f2_get(v[k], lo, hi);
            if (2 * k < n) *p = lo;
            p += HW;
            if (2 * k + 1 < n) *p = hi;
            p += HW;
        }
    }
}

// Zeros that no computed position covers: the words in front of every packed plane and, where positions are mapped into
// another space, that space's padding.  Spread over all CTAs.
__device__ __forceinline__ void fill_zeros(const Args& a, int idx, int threads) {
    if (!a.y) return;
    const int planes = a.k16 >> 2;                           // two per group of 8 channels
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    for (int i = idx; i < planes * a.front; i += threads) {
        const int p = i / a.front, r = i - p * a.front;
        *reinterpret_cast<uint4*>(a.y + (long long)p * a.y_plane - (long long)(r + 1) * 16) = z;
    }
    if (a.map == MAP_SAME) return;
    const Space& d = a.dsp;
    const int rows = d.H + d.pad, wmin = d.split_B ? d.Wf / 2 : d.W, hmin = d.split_B ? d.Hf / 2 : d.H;
    const int right = d.Wp - wmin, per = rows * right + (rows - hmin) * wmin;      // a superset of the padding of a (sub-)image
    const long long n = (long long)d.nimg * per;
    for (long long i = idx; i < n; i += threads) {
        const int img = (int)(i / per);
        int r = (int)(i - (long long)img * per), yy, xx;
        if (r < rows * right) { yy = r / right; xx = wmin + r - yy * right; }
        else { r -= rows * right; yy = hmin + r / wmin; xx = r - (r / wmin) * wmin; }
        bool real = yy < d.H && xx < d.W;
        if (d.split_B) {
            const int p = img / d.split_B;
            real = real && 2 * yy + (p >> 1) < d.Hf && 2 * xx + (p & 1) < d.Wf;
        }
        if (real) continue;
        char* q = a.y + ((long long)img * d.Lp + (long long)yy * d.Wp + xx) * 16;
        for (int p = 0; p < planes; ++p) *reinterpret_cast<uint4*>(q + (long long)p * a.y_plane) = z;
    }
}

// The factors of the epilogue, by its `threads` threads (idx among them; named barrier 1): the bound of the output and with
// it the power of two the packed values are stored at, and per output channel scale and shift with the range scaling of
// input and filter undone.  Returns that power of two.
__device__ __forceinline__ float epilogue_setup(const Args& a, float* s_scale, float* s_bias, unsigned int* words, int idx, int threads, int k0, int n, float comp) {
    // max |x| is one word, or one per block of the packing pass
    unsigned int mx = 0;
    if (a.x_slots > 1) {
        mx = __reduce_max_sync(0xffffffffu, slots_max(a.x_meta + 1, a.x_slots, idx, threads));
        if ((idx & 31) == 0 && mx) atomicMax(&words[0], mx);
    } else mx = __float_as_uint(__ldcg(a.x_meta + 1));
    const float res = a.res ? __ldcg(a.res_meta + 1) : 0.f, inv = 1.f / (__ldcg(a.x_meta) * a.w_meta[0]);
    const float l1 = a.w_meta[1], bmax = a.w_meta[2];
    for (int k = idx; k < n; k += threads) {
        const int oc = k0 + k;
        s_scale[k] = inv * comp * (a.scale && oc < a.K ? __ldg(a.scale + oc) : 1.f);
        s_bias[k] = a.bias && oc < a.K ? __ldg(a.bias + oc) : 0.f;
    }
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
    if (a.x_slots > 1) mx = *(volatile unsigned int*)&words[0];
    const float ys = range_scale(__uint_as_float(mx) * l1 + bmax + res, 15);
    if (a.y_scale && blockIdx.x == 0 && idx == 0) *a.y_scale = ys;
    return ys;
}
// The largest |y| of a CTA: into the tensor's word, or (NCHW outputs) into the CTA's entry of the caller's table.
__device__ __forceinline__ void leave_max(const Args& a, unsigned int m) {
    if (!a.y_slots) return;
    if (a.y_slots_clear) a.y_slots[blockIdx.x] = __uint_as_float(m);
    else if (m) atomicMax(reinterpret_cast<unsigned int*>(a.y_slots), m);
}

// Accumulators of 16 channels -> sums, the range scaling left in (conv_tc.cu: load_chunk explains `comp`).
template <int NT>
__device__ __forceinline__ void load16(const Args& a, uint32_t taddr, float (&v)[16], int blocks) {
    uint32_t r[16], r2[16];
    const float comp = fmaf(a.rz_unit, (float)blocks, 1.f);
    tmem_ld(taddr, r);
    tmem_ld(taddr + NT, r2);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = fmaf(__uint_as_float(r2[k]), 1.f / 2048.f, __uint_as_float(r[k]) * comp);
    if (a.nmain == 2 && blocks > 1) {             // (the second accumulator exists from two blocks on)
        tmem_ld(taddr + 2 * NT, r2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = fmaf(__uint_as_float(r2[k]), comp, v[k]);
    }
}

// ... with scale and shift applied: `scale` carries the compensation, the small accumulator takes scale * `small`.
template <int NT>
__device__ __forceinline__ void scaled16(const Args& a, uint32_t taddr, const float* scale, const float* bias, float small, f2 (&v)[8]) {
    uint32_t r[16], r2[16];
    tmem_ld(taddr, r);
    tmem_ld(taddr + NT, r2);
    const f2 sm = f2_of(small, small);
    f2 s[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(scale + 4 * k), b = *reinterpret_cast<const ulonglong2*>(bias + 4 * k);
        s[2 * k] = t.x; s[2 * k + 1] = t.y;
        v[2 * k] = b.x; v[2 * k + 1] = b.y;
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        v[k] = f2_fma(f2_of(r2[2 * k], r2[2 * k + 1]), f2_mul(s[k], sm), v[k]);
        v[k] = f2_fma(f2_of(r[2 * k], r[2 * k + 1]), s[k], v[k]);
    }
    if (a.nmain == 2 && a.nkb > 1) {
        tmem_ld(taddr + 2 * NT, r2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = f2_fma(f2_of(r2[2 * k], r2[2 * k + 1]), s[k], v[k]);
    }
}

// 2x2 / 2 and 3x3 / 2 maxima of a chunk of 16 channels.  `p`: each lane's largest of its column over the window's rows, not
// negative (the layer has a ReLU).  Neighbouring lanes trade halves, so that the even one ends with the channels 0-7 and the
// odd one with 8-15 of column pair lane / 2.  `next`: those channels of the pair's right column, which the 3x3 window of the
// pair to the right reads.
__device__ __forceinline__ void pool_columns(const f2 (&p)[8], int odd, float (&m)[8], float (&next)[8]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float a0, a1, b0, b1;
        f2_get(p[k], a0, a1);
        f2_get(p[k + 4], b0, b1);
        const float k0 = odd ? b0 : a0, k1 = odd ? b1 : a1;
        const float r0 = __shfl_xor_sync(0xffffffffu, odd ? a0 : b0, 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? a1 : b1, 1);
        m[2 * k] = max_nan(k0, r0); m[2 * k + 1] = max_nan(k1, r1);
        next[2 * k] = odd ? k0 : r0; next[2 * k + 1] = odd ? k1 : r1;
    }
}

// Waits (bounded) for the copies of every stage, by what the producer left: the next stage and its phase.  Stages never used pass at
// once.
__device__ __forceinline__ void copies_landed(uint64_t* full_bar, int ns, unsigned int left) {
    const int st = (int)(left & 255u);
    const uint32_t use = left >> 8 & 1u;
    for (int s = 0; s < ns; ++s) mbar_wait(&full_bar[s], s < st ? use : use ^ 1u);
}

// POOL: the epilogue also does the max pooling that follows.  The feature map of full size — the largest tensor of the network
// at a stem or between VGG's first stages — is then never written nor read back, and the epilogue splits and stores a quarter of
// the values.  Rows meet in registers (the two position tiles are two rows; a 3x3 window's third row stays from the tile before),
// columns by shuffles, and where a 3x3 window reaches into another warp's columns, over shared memory.  What it costs is the
// MMAs of lanes behind the end of a row (configure weighs that).
template <int NT, int MT, int MODE, int POOL = POOL_NONE>
__global__ void __launch_bounds__(PK_THREADS, 1) conv_pk_kernel(const __grid_constant__ Args a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_raw);          // [ns] the copies of a stage have landed
    uint64_t* empty_bar = full_bar + PK_MAXNS;                            // [ns] its MMAs are done
    uint64_t* tfull_bar = empty_bar + PK_MAXNS;                           // [nbuf*MT] a position tile's accumulators are complete
    uint64_t* tempty_bar = tfull_bar + 8;                                 // [nbuf*MT] ... and have been read
    uint64_t* wfull_bar = tempty_bar + 8;                                 // [groups of a tile] the resident filter blocks of a stage have landed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wfull_bar + PK_MAXRES);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned int* words = tmem_slot + 2;                                  // [0] max|x|, [2] max|y| of this CTA, [3] what the producer has asked for
    float* s_scale = reinterpret_cast<float*>(smem_raw + PK_HEADER);
    float* s_bias = s_scale + a.s_floats;
    float* edge = s_bias + a.s_floats;                                    // POOL_3x3: [2][group][warp][2][8] right columns of a warp's last pair
    unsigned char* wfix = reinterpret_cast<unsigned char*>(edge + (POOL == POOL_3x3 ? 512 : 0));      // [wres] the block of output channels' whole filter
    unsigned char* stage0 = wfix + a.wres;
    static_assert(!POOL || MT == 2, "two rows");
    const int below = POOL ? a.sp.Wp : M_TILE;                            // from one position tile to the next
    constexpr int MAXTAPS = MODE == MODE_S2 ? 4 : MODE;
    const uint32_t a_bytes = (uint32_t)a.P * 64u, b_slot = 64u * NT * MAXTAPS;      // of one channel block
    const uint32_t stage_bytes = (uint32_t)a.kps * (a_bytes + (a.wres ? 0u : b_slot));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nbuf = a.nbuf;
    const Walk walk = walk_of<POOL>(a);

    if (tid == 32) {
        for (int s = 0; s < a.ns; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], MT); }
        for (int b = 0; b < 8; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 4 * (NT / 16)); }
        if (a.wres) for (int g = 0; g < PK_MAXRES; ++g) mbar_init(&wfull_bar[g], 1);
        *abort_flag = 0;
        words[0] = words[1] = words[2] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // nothing a kernel before this one in the stream may have written is touched before this (programmatic dependent launch)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            int st = 0, use = 0, loaded = 0;             // loaded: groups of the resident filter asked for
            for (long long t = walk.t; t < walk.end && !*abort_flag; t += walk.step) {
                long long g0; int cnt, ocb, img, pair, seg;
                tile_at<POOL>(a, MT, t, g0, cnt, ocb, img, pair, seg);
                bool ok = true;
                int parity = 0, cb = 0;
                for (int kb0 = 0; kb0 < a.nkb && ok; kb0 += a.kps) {
                    if (!mbar_wait(&empty_bar[st], (uint32_t)(use ^ 1))) { *abort_flag = 1; ok = false; break; }
                    unsigned char* S = stage0 + (size_t)st * stage_bytes;
                    const int n = a.nkb - kb0 < a.kps ? a.nkb - kb0 : a.kps;
                    // (with several blocks per stage every block has the same taps: one-tap filters only)
                    const int rows = M_TILE + (cnt - 1) * below + patch_halo<MODE>(a.sp, parity);
                    const uint32_t run = (uint32_t)rows * 16u, fb = 64u * NT * (uint32_t)taps_of<MODE>(parity);
                    mbar_expect_tx(&full_bar[st], (uint32_t)n * (4u * run + (a.wres ? 0u : fb)));
                    const char* src = a.x + (g0 - patch_shift<MODE>(a.sp, parity) + (MODE == MODE_S2 ? (long long)parity * a.sp.total : 0)) * 16 + (long long)cb * 4 * a.x_plane;
                    if (!a.wres) bulk_g2s(S + (size_t)a.kps * a_bytes, a.wt + filter_offset<MODE, NT>(a, ocb, parity, cb), (uint32_t)n * fb, &full_bar[st]);
                    else if (t == walk.t) {
                        mbar_expect_tx(&wfull_bar[loaded], (uint32_t)n * fb);
                        bulk_g2s(wfix + filter_offset<MODE, NT>(a, 0, parity, cb), a.wt + filter_offset<MODE, NT>(a, ocb, parity, cb), (uint32_t)n * fb, &wfull_bar[loaded]);
                        ++loaded;
                    }
                    for (int k = 0; k < n; ++k) {
                        // planes of a block: (group 0 hi, group 0 lo, group 1 hi, group 1 lo) -> shared [hi: group 0, group 1][lo: group 0, group 1]
                        unsigned char* A = S + (size_t)k * a_bytes;
                        bulk_g2s(A, src, run, &full_bar[st]);
                        bulk_g2s(A + (size_t)a.P * 16, src + 2 * a.x_plane, run, &full_bar[st]);
                        bulk_g2s(A + (size_t)a.P * 32, src + a.x_plane, run, &full_bar[st]);
                        bulk_g2s(A + (size_t)a.P * 48, src + 3 * a.x_plane, run, &full_bar[st]);
                        src += 4 * a.x_plane;
                    }
                    cb += n;
                    if (MODE == MODE_S2 && cb == a.cbl) { cb = 0; ++parity; }
                    if (++st == a.ns) { st = 0; use ^= 1; }
                }
                if (!ok) break;
            }
            words[3] = (unsigned int)(st | use << 8 | loaded << 9);
        }
        __syncwarp();
    } else if (warp < PK_EW0) {
        const int mt = __shfl_sync(0xffffffffu, warp - 1, 0);
        if (mt < MT) {
            long long j = 0;
            int st = 0, use = 0;
            bool here = a.wres == 0;                       // the resident filter has been waited for
            for (long long t = walk.t; t < walk.end && !*abort_flag; t += walk.step, ++j) {
                long long g0; int cnt, ocb, img, pair, seg;
                tile_at<POOL>(a, MT, t, g0, cnt, ocb, img, pair, seg);
                bool ok = true;
                if (mt >= cnt) {               // a smaller tile of the last round: only keep the stages' hand-over in step
                    for (int kb0 = 0; kb0 < a.nkb && ok; kb0 += a.kps) {
                        ok = mbar_wait(&full_bar[st], (uint32_t)use);
                        if (ok && lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty_bar[st])) : "memory");
                        if (++st == a.ns) { st = 0; use ^= 1; }
                    }
                    if (!ok) { *abort_flag = 1; break; }
                    continue;
                }
                const int slot = (nbuf == 2 ? (int)(j & 1) : 0) * MT + mt;
                if (!mbar_wait(&tempty_bar[slot], (uint32_t)(((nbuf == 2 ? j >> 1 : j) & 1) ^ 1))) { *abort_flag = 1; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(slot * a.tile_cols);
                int parity = 0, cb = 0;
                for (int kb0 = 0; kb0 < a.nkb; kb0 += a.kps) {
                    if (!mbar_wait(&full_bar[st], (uint32_t)use) || (!here && !mbar_wait(&wfull_bar[kb0 / a.kps], 0))) { *abort_flag = 1; ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t S = smem_u32(stage0) + (uint32_t)st * stage_bytes;
                    const int kend = kb0 + a.kps < a.nkb ? kb0 + a.kps : a.nkb;
                    const uint32_t fb = 64u * NT * (uint32_t)taps_of<MODE>(parity);
                    const uint32_t F = a.wres ? smem_u32(wfix) + (uint32_t)filter_offset<MODE, NT>(a, 0, parity, cb) : S + (uint32_t)a.kps * a_bytes;
                    if (elect_one()) {
                        for (int kb = kb0; kb < kend; ++kb)
                            pk_issue<NT, MODE>(a, d, S + (uint32_t)(kb - kb0) * a_bytes, F + (uint32_t)(kb - kb0) * fb,
                                               (uint32_t)(mt * below), parity, a.nmain == 2 && (kb & 1), kb < 2 && (kb == 0 || a.nmain == 2));
                        mma_commit(&empty_bar[st]);
                        if (kend == a.nkb) mma_commit(&tfull_bar[slot]);
                    }
                    __syncwarp();
                    cb += kend - kb0;
                    if (MODE == MODE_S2 && cb == a.cbl) { cb = 0; ++parity; }
                    if (++st == a.ns) { st = 0; use ^= 1; }
                }
                if (!ok) break;
                here = true;
            }
        }
    } else {
        const int e = tid - PK_EW0 * 32, grp = (warp - PK_EW0) >> 2, q = warp & 3;
        const float comp = fmaf(a.rz_unit, (float)a.nkb, 1.f), small = 1.f / (2048.f * comp);
        const float ys = epilogue_setup(a, s_scale, s_bias, words, e, PK_EPI, 0, a.s_floats, comp);
        fill_zeros(a, (int)blockIdx.x * PK_EPI + e, (int)gridDim.x * PK_EPI);
        constexpr int CHUNKS = NT / 16;
        const int k_end = a.nchw ? a.K : a.k16;            // channels that are stored anywhere
        float ymax = 0.f;
        long long j = 0;
        if constexpr (POOL != POOL_NONE) {
            static_assert(POOL != POOL_3x3 || CHUNKS <= PK_GROUPS, "a group keeps one chunk's row above");
            f2 above[8];                                   // the lower row of the tile before
#pragma unroll
            for (int k = 0; k < 8; ++k) above[k] = 0ull;
            const int odd = lane & 1;
            // (with 3x3 windows the four warps of a group stay together: they leave the loop by the vote below)
            for (long long t = walk.t; grp < CHUNKS && t < walk.end && (POOL == POOL_3x3 || !*abort_flag); ++t, ++j) {
                long long g0; int cnt, ocb, img, pair, seg;
                tile_at<POOL>(a, MT, t, g0, cnt, ocb, img, pair, seg);
                const int slot = nbuf == 2 ? 2 * (int)(j & 1) : 0, x = seg * M_TILE + q * 32 + lane;
                const uint32_t phase = (uint32_t)((nbuf == 2 ? j >> 1 : j) & 1);
                const bool upper = x < a.sp.W, lower = upper && 2 * pair + 1 < a.sp.H;
                Where w;
                w.same = g0; w.in = false;
                w.valid = t >= walk.first && (x >> 1) < a.dsp.W;
                w.out = (long long)img * a.dsp.Lp + (long long)pair * a.dsp.Wp + (x >> 1);
                const bool ok = __all_sync(0xffffffffu, mbar_wait(&tfull_bar[slot], phase) && mbar_wait(&tfull_bar[slot + 1], phase));
                if (!ok) *abort_flag = 1;
                if (POOL != POOL_3x3 && !ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int chunk = grp; chunk < CHUNKS; chunk += PK_GROUPS) {
                    const int k0 = chunk * 16;
                    const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(slot * a.tile_cols + k0);
                    const bool act = ok && k0 < k_end;
                    f2 v[8], p[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) p[k] = POOL == POOL_3x3 && pair > 0 ? above[k] : 0ull;
                    // largest of each column, and of zero
                    auto rows = [&](bool real) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            float a0, a1, b0, b1;
                            if (!real) v[k] = 0ull;
                            f2_get(v[k], a0, a1);
                            f2_get(p[k], b0, b1);
                            p[k] = f2_of(max_nan(a0, b0), max_nan(a1, b1));
                        }
                    };
                    if (act) {
                        scaled16<NT>(a, at, s_scale + k0, s_bias + k0, small, v);
                        rows(upper);
                        scaled16<NT>(a, at + (uint32_t)a.tile_cols, s_scale + k0, s_bias + k0, small, v);
                        rows(lower);
                        if (POOL == POOL_3x3) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                float b0, b1;
                                f2_get(v[k], b0, b1);
                                above[k] = f2_of(max_nan(b0, 0.f), max_nan(b1, 0.f));
                            }
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane < 2) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty_bar[slot + lane])) : "memory");
                    float m[8], next[8];
                    pool_columns(p, odd, m, next);
                    if constexpr (POOL == POOL_3x3) {
                        float* mine = edge + (((int)(j & 1) * PK_GROUPS + grp) * 4 + q) * 16 + odd * 8;
                        if (lane >= 30) {
                            *reinterpret_cast<float4*>(mine) = make_float4(next[0], next[1], next[2], next[3]);
                            *reinterpret_cast<float4*>(mine + 4) = make_float4(next[4], next[5], next[6], next[7]);
                        }
#pragma unroll
                        for (int k = 0; k < 8; ++k) next[k] = __shfl_up_sync(0xffffffffu, next[k], 2);
                        uint32_t bad = (!ok || *abort_flag) ? 1u : 0u;
                        asm volatile("{\n\t.reg .pred in, out;\n\tsetp.ne.u32 in, %0, 0;\n\tbarrier.cta.red.or.pred out, %1, 128, in;\n\tselp.u32 %0, 1, 0, out;\n\t}" : "+r"(bad) : "r"(2 + grp) : "memory");
                        if (bad) { j = -1; break; }
                        if (lane < 2) {
                            const float* left = mine - 16;
#pragma unroll
                            for (int k = 0; k < 8; ++k) next[k] = q > 0 ? left[k] : 0.f;
                        }
#pragma unroll
                        for (int k = 0; k < 8; ++k) m[k] = max_nan(m[k], next[k]);
                    }
                    if (k0 >= k_end) continue;
                    f2 out[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) out[k] = f2_of(m[2 * k], m[2 * k + 1]);
                    store(a, w, k0 + 8 * odd, out, ys, ymax);
                }
                if (j < 0) break;
            }
        } else
        for (long long t = walk.t; t < walk.end && !*abort_flag; t += walk.step, ++j) {
            long long g0; int cnt, ocb;
            pk_tile_of(a, MT, t, g0, cnt, ocb);
            // Two groups to each of two position tiles, or all four to one: where a position goes is worked out once for
            // all of a group's chunks of channels.  (A last tile without its second position tile leaves two groups idle: they
            // have not followed the first one's barriers, whose parity alone would tell them nothing.)
            const int mt = MT == 2 ? grp >> 1 : 0, first = MT == 2 ? grp & 1 : grp, step = MT == 2 ? 2 : PK_GROUPS;
            if (mt >= cnt || first >= CHUNKS) continue;
            const int slot = (nbuf == 2 ? (int)(j & 1) : 0) * MT + mt;
            const Where w = place(a, g0 + mt * M_TILE + q * 32 + lane);
            bool waited = false, ok = true;
#pragma unroll 1
            for (int chunk = first; chunk < CHUNKS; chunk += step) {
                const int k0 = ocb * NT + chunk * 16;
                f2 rv[8], v[8];
                if (a.res) residual(a, w.same, w.valid, k0, rv);          // in flight while the accumulators are waited for
                if (!waited) {
                    if (!mbar_wait(&tfull_bar[slot], (uint32_t)((nbuf == 2 ? j >> 1 : j) & 1))) { *abort_flag = 1; ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    waited = true;
                }
                if (k0 < k_end) scaled16<NT>(a, tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(slot * a.tile_cols + chunk * 16), s_scale + k0, s_bias + k0, small, v);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty_bar[slot])) : "memory");
                if (k0 >= k_end) continue;
                if (a.res) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = f2_add(v[k], rv[k]);
                }
                store(a, w, k0, v, ys, ymax);
            }
            if (!ok) break;
        }
        const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(ymax));
        if (lane == 0) atomicMax(&words[2], m);
    }

    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
        if (*abort_flag) {
            if (a.status) atomicCAS(a.status, 0, 1);
            // leaving early, whoever gave up: no copy of this CTA may still be in flight when it exits
            copies_landed(full_bar, a.ns, words[3]);
            for (int g = 0; g < (int)(words[3] >> 9); ++g) mbar_wait(&wfull_bar[g], 0);
        }
        if (a.status && words[2] >= 0x7f800000u) atomicCAS(a.status, 0, 2);      // an output that is not finite
        leave_max(a, words[2]);
    }
    if (a.y_slots && blockIdx.x == 0)
        for (int i = gridDim.x + tid; i < a.y_slots_clear; i += PK_THREADS) a.y_slots[i] = 0.f;
    if (warp == 3) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
}

// Small batches: too few tiles to fill the chip, and the chain of channel blocks of a tile is the time.  The `ksplit` CTAs
// of a cluster share one tile of 128 positions x NT output channels, each accumulating `kb_per` channel blocks; every CTA
// then owns 128 / ksplit of the positions, receives the ranks' partial sums of them through distributed shared memory and
// adds them in rank order.  One tile per CTA, 256 threads and at most half of an SM's shared memory, so that the next
// launch's CTAs set up beside this one's and have their first filter blocks in shared memory when griddepcontrol.wait
// returns (the filter is no earlier kernel's output).
constexpr int SPLIT_THREADS = 256, SPLIT_EPI = 128;

template <int NT, int MODE>
__global__ void __launch_bounds__(SPLIT_THREADS, 2) conv_pk_split_kernel(const __grid_constant__ Args a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_raw);
    uint64_t* empty_bar = full_bar + PK_MAXNS;
    uint64_t* tfull_bar = empty_bar + PK_MAXNS;
    uint64_t* xfull_bar = tfull_bar + 1;                                  // the ranks' partial sums of this CTA's positions have arrived
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xfull_bar + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned int* words = tmem_slot + 2;
    constexpr int XROW = NT + 4;                                          // floats per row of the exchange buffer
    float* s_scale = reinterpret_cast<float*>(smem_raw + 256);            // [NT] of this block's channels
    float* s_bias = s_scale + NT;
    float* xbuf = reinterpret_cast<float*>(smem_raw + PK_HEADER);         // [ksplit][128 / ksplit][XROW]
    unsigned char* stage0 = reinterpret_cast<unsigned char*>(xbuf) + (a.ksplit > 1 ? 128 * XROW * 4 : 0);
    constexpr int MAXTAPS = MODE == MODE_S2 ? 4 : MODE;
    const uint32_t a_bytes = (uint32_t)a.P * 64u, b_slot = 64u * NT * MAXTAPS;
    const uint32_t stage_bytes = (uint32_t)a.kps * (a_bytes + b_slot);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ks = a.ksplit, rank = (int)blockIdx.x % ks, tile = (int)blockIdx.x / ks;
    const int ocb = tile % a.n_ocb;
    const long long g0 = (long long)(tile / a.n_ocb) * M_TILE;
    const int kb_lo = rank * a.kb_per, kb_hi = kb_lo + a.kb_per < a.nkb ? kb_lo + a.kb_per : a.nkb;
    const int used = (a.nkb + a.kb_per - 1) / a.kb_per;                   // ranks that have a channel block (the others only finish positions)

    if (tid == 32) {
        for (int s = 0; s < a.ns; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(tfull_bar, 1);
        mbar_init(xfull_bar, 1);
        *abort_flag = 0;
        words[0] = words[1] = words[2] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // every CTA of the cluster runs before its shared memory is written from outside (waited for ahead of the exchange)
    if (ks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            // parity and block of channel block kb (MODE_S2; parity 0 otherwise)
            auto parity_of = [&](int kb) { return MODE == MODE_S2 ? kb / a.cbl : 0; };
            auto announce = [&](int kb0, int st) {                         // bytes of the stage, and its filter blocks
                const int p = parity_of(kb0), cb = kb0 - p * a.cbl, n = kb_hi - kb0 < a.kps ? kb_hi - kb0 : a.kps;
                const uint32_t run = (uint32_t)(M_TILE + patch_halo<MODE>(a.sp, p)) * 16u, fb = 64u * NT * (uint32_t)taps_of<MODE>(p);
                mbar_expect_tx(&full_bar[st], (uint32_t)n * (4u * run + fb));
                bulk_g2s(stage0 + (size_t)st * stage_bytes + (size_t)a.kps * a_bytes, a.wt + filter_offset<MODE, NT>(a, ocb, p, cb), (uint32_t)n * fb, &full_bar[st]);
            };
            auto patch = [&](int kb0, int st) {
                const int p = parity_of(kb0), cb = kb0 - p * a.cbl, n = kb_hi - kb0 < a.kps ? kb_hi - kb0 : a.kps;
                const uint32_t run = (uint32_t)(M_TILE + patch_halo<MODE>(a.sp, p)) * 16u;
                const char* src = a.x + (g0 - patch_shift<MODE>(a.sp, p) + (MODE == MODE_S2 ? (long long)p * a.sp.total : 0)) * 16 + (long long)cb * 4 * a.x_plane;
                for (int k = 0; k < n; ++k) {
                    unsigned char* A = stage0 + (size_t)st * stage_bytes + (size_t)k * a_bytes;
                    bulk_g2s(A, src, run, &full_bar[st]);
                    bulk_g2s(A + (size_t)a.P * 16, src + 2 * a.x_plane, run, &full_bar[st]);
                    bulk_g2s(A + (size_t)a.P * 32, src + a.x_plane, run, &full_bar[st]);
                    bulk_g2s(A + (size_t)a.P * 48, src + 3 * a.x_plane, run, &full_bar[st]);
                    src += 4 * a.x_plane;
                }
            };
            int st = 0;
            for (int kb0 = kb_lo; kb0 < kb_hi && st < a.ns; kb0 += a.kps, ++st) announce(kb0, st);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            int use = 0, n = 0;
            st = 0;
            for (int kb0 = kb_lo; kb0 < kb_hi; kb0 += a.kps, ++n) {
                if (n >= a.ns) {
                    if (!mbar_wait(&empty_bar[st], (uint32_t)(use ^ 1))) { *abort_flag = 1; break; }
                    announce(kb0, st);
                }
                patch(kb0, st);
                if (++st == a.ns) { st = 0; use ^= 1; }
            }
            words[4] = (unsigned int)(st | use << 8);
        }
        __syncwarp();
    } else if (warp == 1) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        int st = 0, use = 0;
        for (int kb0 = kb_lo; kb0 < kb_hi; kb0 += a.kps) {
            if (!mbar_wait(&full_bar[st], (uint32_t)use)) { *abort_flag = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t S = smem_u32(stage0) + (uint32_t)st * stage_bytes;
            const int kend = kb0 + a.kps < kb_hi ? kb0 + a.kps : kb_hi, parity = MODE == MODE_S2 ? kb0 / a.cbl : 0;
            const uint32_t fb = 64u * NT * (uint32_t)taps_of<MODE>(parity);
            if (elect_one()) {
                for (int kb = kb0; kb < kend; ++kb) {
                    const int kr = kb - kb_lo;
                    pk_issue<NT, MODE>(a, tmem, S + (uint32_t)(kb - kb0) * a_bytes, S + (uint32_t)a.kps * a_bytes + (uint32_t)(kb - kb0) * fb, 0u, parity,
                                       a.nmain == 2 && (kr & 1), kr < 2 && (kr == 0 || a.nmain == 2));
                }
                mma_commit(&empty_bar[st]);
                if (kend == kb_hi) mma_commit(tfull_bar);
            }
            __syncwarp();
            if (++st == a.ns) { st = 0; use ^= 1; }
        }
    } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    // All eight warps drain tensor memory (warps w and w + 4 share a lane quarter and take every other chunk of channels)
    // and finish positions; the last four have set up the factors meanwhile.
    const int q = warp & 3, rpc = 128 / ks;                               // rpc: positions each CTA of the cluster finishes
    float* ys_word = reinterpret_cast<float*>(words + 3);
    const float comp = fmaf(a.rz_unit, (float)a.nkb, 1.f), small = 1.f / (2048.f * comp);      // (one CTA per tile)
    if (warp >= 4) {
        const int e = tid - 128;
        const float ys = epilogue_setup(a, s_scale, s_bias, words, e, SPLIT_EPI, ocb * NT, NT, ks == 1 ? comp : 1.f);      // for this block's channels
        if (e == 0) {
            *ys_word = ys;
            if (ks > 1) mbar_expect_tx(xfull_bar, (uint32_t)(used * rpc * NT * 4));
        }
        fill_zeros(a, (int)blockIdx.x * SPLIT_EPI + e, (int)gridDim.x * SPLIT_EPI);
    }
    __syncwarp();
    __syncthreads();
    const float ys = *ys_word;
    float ymax = 0.f;
    const int k_end = a.nchw ? a.K : a.k16;
    if (ks == 1) {
        const Where w = place(a, g0 + q * 32 + lane);
        const bool ok = mbar_wait(tfull_bar, 0);
        if (!ok) *abort_flag = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (ok)
            for (int c0 = (warp >> 2) * 16; c0 < NT && ocb * NT + c0 < k_end; c0 += 32) {
                f2 rv[8], v[8];
                if (a.res) residual(a, w.same, w.valid, ocb * NT + c0, rv);
                scaled16<NT>(a, tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, s_scale + c0, s_bias + c0, small, v);
                if (a.res) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = f2_add(v[k], rv[k]);
                }
                store(a, w, ocb * NT + c0, v, ys, ymax);
            }
    } else {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank < used) {
            const bool ok = mbar_wait(tfull_bar, 0);
            if (!ok) *abort_flag = 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok) {
                // every value travels with its count of bytes to the owner's barrier: an owner waits for its own
                // positions only, not for the whole cluster
                const int row = q * 32 + lane, owner = row / rpc;
                uint32_t dst, bar;
                const uint32_t mine = smem_u32(xbuf + ((long long)rank * rpc + (row - owner * rpc)) * XROW);
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(mine), "r"(owner));
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_u32(xfull_bar)), "r"(owner));
#pragma unroll 1
                for (int c0 = (warp >> 2) * 16; c0 < NT; c0 += 32) {
                    float v[16];
                    load16<NT>(a, tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v, kb_hi - kb_lo);
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4)
                        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                                     ::"r"(dst + (uint32_t)(c0 + 4 * k4) * 4u), "f"(v[4 * k4]), "f"(v[4 * k4 + 1]), "f"(v[4 * k4 + 2]), "f"(v[4 * k4 + 3]), "r"(bar) : "memory");
                }
            }
        }
        // 8 channels of one position at a time; the residual is in flight while the sums are waited for
        const int u0 = tid, cn = NT / 8;
        auto finish = [&](int u, bool first) {
            const int chunk = u / rpc, lr = u - chunk * rpc, c0 = chunk * 8;       // neighbouring threads: neighbouring positions
            const bool some = u < rpc * cn && ocb * NT + c0 < k_end;
            Where w{};
            f2 rv[4], v[4];
            if (some) {
                w = place(a, g0 + rank * rpc + lr);
                if (a.res) residual(a, w.same, w.valid, ocb * NT + c0, rv);
            }
            if (first && !mbar_wait(xfull_bar, 0)) *abort_flag = 1;
            if (!some) return;
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = 0ull;
            for (int r = 0; r < used; ++r) {
                const ulonglong2* p = reinterpret_cast<const ulonglong2*>(xbuf + ((long long)r * rpc + lr) * XROW + c0);
                const ulonglong2 s = p[0], t = p[1];
                v[0] = f2_add(v[0], s.x); v[1] = f2_add(v[1], s.y); v[2] = f2_add(v[2], t.x); v[3] = f2_add(v[3], t.y);
            }
            const f2* sc = reinterpret_cast<const f2*>(s_scale + c0);
            const f2* bi = reinterpret_cast<const f2*>(s_bias + c0);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = f2_fma(v[k], sc[k], bi[k]);
                if (a.res) v[k] = f2_add(v[k], rv[k]);
            }
            store(a, w, ocb * NT + c0, v, ys, ymax);
        };
        finish(u0, true);
        for (int u = u0 + SPLIT_THREADS; u < rpc * cn; u += SPLIT_THREADS) finish(u, false);
    }
    const unsigned int top = __reduce_max_sync(0xffffffffu, __float_as_uint(ymax));
    if (lane == 0 && top) atomicMax(&words[2], top);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {                                                    // (uniform: nobody writes it behind the barrier)
        if (tid == 0) {
            if (a.status) atomicCAS(a.status, 0, 1);
            copies_landed(full_bar, a.ns, words[4]);
        }
        // The others of the cluster may still be sending to this CTA: it leaves when they have sent (or have left themselves; their
        // waits are bounded like these) and what they sent has landed.
        if (ks > 1) {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (tid == 0) mbar_wait(xfull_bar, 0);
        }
    }
    if (tid == 0) {
        if (a.status && words[2] >= 0x7f800000u) atomicCAS(a.status, 0, 2);
        leave_max(a, words[2]);
    }
    if (a.y_slots && blockIdx.x == 0)
        for (int i = gridDim.x + tid; i < a.y_slots_clear; i += SPLIT_THREADS) a.y_slots[i] = 0.f;
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
}

}  // namespace tdc_pk
