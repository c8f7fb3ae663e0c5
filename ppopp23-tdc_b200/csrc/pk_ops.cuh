// The passes between convolutions on packed activations (pk.h): packing an NCHW input, pooling, BatchNorm + ReLU, and the
// classifier head.  All of them are memory-bound: a thread takes one position and 8 channels, neighbouring threads take
// neighbouring positions, so that every load and store instruction of a warp covers whole lines.
#pragma once
#include "conv_pk.cuh"

namespace tdc_pk {

constexpr int OPS_THREADS = 512;

// What earlier launches of the stream wrote is read by plain loads (or past L1), never by __ldg, which the compiler may move
// ahead of this: the launch may have started before they ended.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Largest value of a block (bit patterns); every thread gets it.
__device__ __forceinline__ unsigned int block_max(unsigned int m, unsigned int* word) {
    if (threadIdx.x == 0) *word = 0;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(word, m);
    __syncthreads();
    m = *word;
    __syncthreads();
    return m;
}

constexpr int PACK_ITEMS = 4;
enum PackKind { PACK_SAME = 0, PACK_SPLIT = 1, PACK_S2D = 2, PACK_ROW3 = 3 };

struct PackArgs {
    const float* x;                       // [B][C][H][W]
    int B, C, H, W;
    const float* absmax; int absmax_n;    // partial maxima of |x|, or nullptr: the range is sampled
    char* y; long long y_plane; int groups, front;
    Space d;
    float* y_scale; float* y_slots;       // the partial maxima of what it wrote, one per block
    float* zero; int zeros;               // the other tensors' meta blocks, cleared here (this is the first launch of a run)
    int* status;                          // 2 where a value does not fit
    uint32_t sample_step;                 // a 1536th of x, rounded up: one value of each such piece is sampled
};

// NCHW -> packed planes.
//   SAME   channels as they are; SPLIT  the same, positions by parity;
//   S2D    channel 4 c + 2 (row parity) + (column parity) of half-size images: a 7x7 stride-2 filter is a 4x4 stride-1 one on
//          these (12 of 16 channels used for an RGB image, one channel block);
//   ROW3   channel 3 c + dx holds column x + dx - 1: a 3x3 filter over few channels is three row taps on these, one channel
//          block where the plain form takes nine taps of a block that is mostly zeros.
// Bound by memory: 4 bytes read and 4 written per value.
//
// EXACT: the sample's place is taken by the true maximum.  Launched in clusters of PACK_CLUSTER, each of which finds the true maximum of x for itself, every CTA of a share of it;
// the second reading comes out of cache.  For inputs of up to PACK_EXACT values that costs about what the round trip of the sample does,
// and layers of that size ran on fp32 arithmetic, which has no range, before they ran on packed operands.
constexpr int PACK_CLUSTER = 8;
constexpr long long PACK_EXACT = 1 << 18;

// Largest magnitude of x[0, n), by the cluster; every thread gets it.
__device__ __forceinline__ unsigned int cluster_absmax(const float* x, long long n, unsigned int* word, unsigned int* peers) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // every CTA runs before its shared memory is written to
    uint32_t rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int first = (int)rank * OPS_THREADS + (int)threadIdx.x;
    constexpr int STEP = PACK_CLUSTER * OPS_THREADS;
    unsigned int m = 0;
    auto take = [&](float v) { m = max(m, __float_as_uint(v) & 0x7fffffffu); };
    const int n4 = reinterpret_cast<uintptr_t>(x) % 16 == 0 ? (int)(n / 4) : 0;      // (n is at most PACK_EXACT)
#pragma unroll 8
    for (int i = first; i < n4; i += STEP) {
        const float4 v = reinterpret_cast<const float4*>(x)[i];
        take(v.x); take(v.y); take(v.z); take(v.w);
    }
#pragma unroll 4
    for (int i = 4 * n4 + first; i < (int)n; i += STEP) take(x[i]);
    m = block_max(m, word);
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (threadIdx.x < PACK_CLUSTER) {
        uint32_t dst;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_u32(peers + rank)), "r"(threadIdx.x));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst), "r"(m) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int k = 0; k < PACK_CLUSTER; ++k) m = max(m, peers[k]);
    return m;
}

// The partial maxima of x, in the form a caller would give them: for larger inputs that want the true one (the clusters' readings add
// up: at a million values they would cost 15 us, this pass costs one launch and one reading).
__global__ void __launch_bounds__(OPS_THREADS) range_kernel(const float* x, long long n, float* slots, int n_slots) {
    __shared__ unsigned int word;
    pdl_enter();
    unsigned int m = 0;
    const long long step = (long long)gridDim.x * OPS_THREADS;
    long long i = (long long)blockIdx.x * OPS_THREADS + threadIdx.x;
    if (reinterpret_cast<uintptr_t>(x) % 16 == 0) {
        const long long n4 = n / 4;
#pragma unroll 4
        for (; i < n4; i += step) {
            const float4 v = reinterpret_cast<const float4*>(x)[i];
            m = max(max(m, __float_as_uint(v.x) & 0x7fffffffu), __float_as_uint(v.y) & 0x7fffffffu);
            m = max(max(m, __float_as_uint(v.z) & 0x7fffffffu), __float_as_uint(v.w) & 0x7fffffffu);
        }
        i = 4 * n4 + (long long)blockIdx.x * OPS_THREADS + threadIdx.x;
    }
    for (; i < n; i += step) m = max(m, __float_as_uint(x[i]) & 0x7fffffffu);
    m = block_max(m, &word);
    if (threadIdx.x == 0) slots[blockIdx.x] = __uint_as_float(m);
    if (blockIdx.x == 0)
        for (int k = (int)gridDim.x + threadIdx.x; k < n_slots; k += OPS_THREADS) slots[k] = 0.f;
}

template <int KIND, bool EXACT>
__global__ void __launch_bounds__(OPS_THREADS, 2) pack_kernel(const PackArgs a) {
    __shared__ unsigned int word, peers[PACK_CLUSTER];
    pdl_enter();
    // the power of two the values are stored at: from the given maxima, the true one, or from 1536 values spread over x, which leaves a
    // factor of 256 for what the sample missed (what lies beyond is reported: the true maximum is known at the end, and the
    // convolution's outputs are NaN).  One value of each 1536th of x, at an offset that goes round by the golden ratio: at a fixed
    // one a batch of 16 images of 3 x 224 x 224 was sampled in one column.
    const long long n = (long long)a.B * a.C * a.H * a.W;
    unsigned int m = 0;
    if (a.absmax) m = slots_max(a.absmax, a.absmax_n, threadIdx.x, OPS_THREADS);
    else if (EXACT) m = cluster_absmax(a.x, n, &word, peers);
    else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint32_t j = threadIdx.x + i * OPS_THREADS;
            const unsigned long long k = (unsigned long long)j * a.sample_step + __umulhi(j * 2654435769u, a.sample_step);
            if (k < (unsigned long long)n) m = max(m, __float_as_uint(a.x[k]) & 0x7fffffffu);
        }
    }
    const float s = range_scale(__uint_as_float(block_max(m, &word)), a.absmax || EXACT ? 14 : 8);
    const uint32_t span = (uint32_t)(a.front + a.d.total), items = span * (uint32_t)a.groups, stride = gridDim.x * OPS_THREADS;
    const int HW = a.H * a.W;                      // (the host keeps an image's plane below 2^31)
    // the 8 values of item i, zeros where it is padding
    auto load = [&](uint32_t i, float (&v)[8]) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 0.f;
        const uint32_t cg = i / span;
        const int g = (int)(i - cg * span) - a.front;
        if (g < 0) return;
        const uint32_t img = fastdiv((uint32_t)g, a.d.fd_Lp), rem = (uint32_t)g - img * (uint32_t)a.d.Lp;
        const int yy = (int)fastdiv(rem, a.d.fd_Wp), xx = (int)rem - yy * a.d.Wp;
        if (yy >= a.d.H || xx >= a.d.W) return;
        const int c0 = (int)cg * 8;
        if (KIND == PACK_SAME || KIND == PACK_SPLIT) {
            int b = (int)img, fy = yy, fx = xx;
            if (KIND == PACK_SPLIT) {
                const int p = b >= 2 * a.B ? 2 : 0, px = b >= (p + 1) * a.B ? 1 : 0;
                b -= (p + px) * a.B; fy = 2 * yy + (p >> 1); fx = 2 * xx + px;
                if (fy >= a.H || fx >= a.W) return;
            }
            const float* xp = a.x + ((long long)b * a.C + c0) * HW + fy * a.W + fx;
#pragma unroll
            for (int k = 0; k < 8; ++k) { if (c0 + k < a.C) v[k] = *xp; xp += HW; }
        } else if (KIND == PACK_S2D) {
            const float* xp = a.x + ((long long)img * a.C + (c0 >> 2)) * HW + 2 * yy * a.W + 2 * xx;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if ((c0 + k) >> 2 < a.C && 2 * yy + ((k >> 1) & 1) < a.H && 2 * xx + (k & 1) < a.W) v[k] = *(xp + (k >> 2) * HW + ((k >> 1) & 1) * a.W + (k & 1));
        } else {
            const float* xp = a.x + (long long)img * a.C * HW + yy * a.W + xx - 1;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = (c0 + k) / 3, dx = (c0 + k) % 3, fx = xx + dx - 1;
                if (c < a.C && fx >= 0 && fx < a.W) v[k] = *(xp + c * HW + dx);
            }
        }
    };
    float big = 0.f;
    auto store = [&](uint32_t i, const float (&v)[8]) {
        const uint32_t cg = i / span;
        const int g = (int)(i - cg * span) - a.front;
#pragma unroll
        for (int k = 0; k < 4; ++k) big = max3_abs(big, v[2 * k], v[2 * k + 1]);
        f2 pv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) pv[k] = f2_of(v[2 * k], v[2 * k + 1]);
        uint4 hi, lo;
        split8(pv, s, hi, lo);
        char* p = a.y + (long long)cg * 2 * a.y_plane + (long long)g * 16;
        *reinterpret_cast<uint4*>(p) = hi;
        *reinterpret_cast<uint4*>(p + a.y_plane) = lo;
    };
    // PACK_ITEMS at a time: 32 loads in flight per thread
    uint32_t i = blockIdx.x * OPS_THREADS + threadIdx.x;
    for (; i + (PACK_ITEMS - 1) * stride < items; i += PACK_ITEMS * stride) {
        float v[PACK_ITEMS][8];
#pragma unroll
        for (int k = 0; k < PACK_ITEMS; ++k) load(i + k * stride, v[k]);
#pragma unroll
        for (int k = 0; k < PACK_ITEMS; ++k) store(i + k * stride, v[k]);
    }
    for (; i < items; i += 2 * stride) {
        float v[8], w[8];
        const bool two = i + stride < items;
        load(i, v);
        if (two) load(i + stride, w);
        store(i, v);
        if (two) store(i + stride, w);
    }
    const unsigned int most = block_max(__float_as_uint(big), &word);
    if (threadIdx.x == 0) {
        a.y_slots[blockIdx.x] = __uint_as_float(most);
        if (blockIdx.x == 0) *a.y_scale = s;
        if (a.status && !(__uint_as_float(most) * s < 65520.f)) atomicCAS(a.status, 0, 2);       // (from there on a value rounds to infinity)
    }
    if (blockIdx.x == 0)
        for (int k = threadIdx.x; k < a.zeros; k += OPS_THREADS) a.zero[k] = 0.f;
}

constexpr int POOL_THREADS = 256;

struct PoolArgs {
    const float* x; long long x_plane; Space sp;       // fp32 planes
    const float* x_max;                                // [1] max |x|
    int C, k, stride, pad;                             // max pooling; mode AFFINE: k = stride = 1 or 2 (average of k x k)
    const float* scale; const float* shift;            // mode AFFINE: relu(x * scale[c] + shift[c]) before the average
    const float* bound;                                // mode AFFINE: {max |scale|, max |shift|}
    char* y; long long y_plane; int front;             // packed output, or nullptr
    float* yf; long long yf_plane;                     // fp32 planes, or nullptr
    Space d;
    float* y_scale; float* y_max;                      // y_scale: nullptr where an existing tensor is written into
};

// Items (positions) a thread has in flight: eight to eighteen 16-byte loads.
template <int K> struct PoolItems { static constexpr int N = K == 1 ? 4 : (K == 2 ? 2 : 1); };

// fp32 planes -> packed and / or fp32 planes of a smaller or equal image: max pooling, or BatchNorm + ReLU (+ 2x2 average).
// `K`: the window (0: taken from the arguments).  Bound by memory.  A block works on one group of 8 channels (blockIdx.y), so
// its scale and shift are loaded once, and with a compile-time window all loads of a thread's items are in flight at once.
template <bool AFFINE, int K>
__global__ void __launch_bounds__(POOL_THREADS, K == 1 ? 3 : 2) pool_pk_kernel(const __grid_constant__ PoolArgs a) {
    __shared__ unsigned int word;
    constexpr int N = PoolItems<K>::N, W = K > 0 ? K * K : 1;
    const int cg = (int)blockIdx.y, c0 = cg * 8;
    const bool some = c0 < a.C, two = c0 + 4 < a.C;
    float sc[8], sh[8];
    if (AFFINE) {
#pragma unroll
        for (int k = 0; k < 8; ++k) { const bool has = c0 + k < a.C; sc[k] = has ? __ldg(a.scale + c0 + k) : 0.f; sh[k] = has ? __ldg(a.shift + c0 + k) : 0.f; }
    }
    if (threadIdx.x == 0) word = 0;
    pdl_enter();
    __syncthreads();
    float bound = __ldcg(a.x_max);
    if (AFFINE) bound = bound * a.bound[0] + a.bound[1];
    const float s = range_scale(bound, 15), none = AFFINE ? 0.f : -INFINITY;
    const float* xg = a.x + (long long)(cg * 2) * a.x_plane;
    char* yg = a.y + (long long)cg * 2 * a.y_plane;
    float* fg = a.yf + (long long)(cg * 2) * a.yf_plane;
    const int end = (int)a.d.total, step = (int)gridDim.x * POOL_THREADS;
    float big = 0.f;
    for (int g0 = (int)(blockIdx.x * POOL_THREADS + threadIdx.x) - a.front; g0 < end; g0 += N * step) {
        float4 t[N][W], u[N][W];
        bool real[N];
        const float* base[N];
        int y0[N], x0[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int g = g0 + n * step;
            real[n] = false;
            base[n] = xg; y0[n] = x0[n] = 0;
            if (g >= 0 && g < end && some) {
                const uint32_t img = fastdiv((uint32_t)g, a.d.fd_Lp), rem = (uint32_t)g - img * (uint32_t)a.d.Lp;
                const int oy = (int)fastdiv(rem, a.d.fd_Wp), ox = (int)rem - oy * a.d.Wp;
                real[n] = oy < a.d.H && ox < a.d.W;
                y0[n] = oy * a.stride - a.pad; x0[n] = ox * a.stride - a.pad;
                base[n] = xg + ((long long)img * a.sp.Lp + (long long)y0[n] * a.sp.Wp + x0[n]) * 4;      // (only formed, never read, where outside)
            }
            if constexpr (K > 0) {
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    t[n][w] = u[n][w] = make_float4(none, none, none, none);
                    if (real[n] && (unsigned)(y0[n] + w / K) < (unsigned)a.sp.H && (unsigned)(x0[n] + w % K) < (unsigned)a.sp.W) {
                        const float* p = base[n] + ((w / K) * a.sp.Wp + w % K) * 4;
                        t[n][w] = *reinterpret_cast<const float4*>(p);
                        if (two) u[n][w] = *reinterpret_cast<const float4*>(p + a.x_plane);
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int g = g0 + n * step;
            if (g >= end) break;
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = none;
            auto take = [&](const float4& p, const float4& q) {
                const float in[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (AFFINE) v[k] += max_nan(fmaf(in[k], sc[k], sh[k]), 0.f);
                    else v[k] = max_nan(v[k], in[k]);
                }
            };
            if constexpr (K > 0) {
                if constexpr (AFFINE || W % 2 == 0) {
#pragma unroll
                    for (int w = 0; w < W; ++w) take(t[n][w], u[n][w]);
                } else {
                    // three operands at a time
#pragma unroll
                    for (int w = 0; w < W; w += 2) {
                        const float4 &p = t[n][w], &q = u[n][w], &r = t[n][w + 1 < W ? w + 1 : w], &s4 = u[n][w + 1 < W ? w + 1 : w];
                        const float x[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w}, y[8] = {r.x, r.y, r.z, r.w, s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                        for (int k = 0; k < 8; ++k) asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(v[k]) : "f"(x[k]), "f"(y[k]));
                    }
                }
            } else if (real[n]) {
                for (int dy = 0; dy < a.k; ++dy)
                    for (int dx = 0; dx < a.k; ++dx) {
                        if ((unsigned)(y0[n] + dy) >= (unsigned)a.sp.H || (unsigned)(x0[n] + dx) >= (unsigned)a.sp.W) continue;
                        const float* p = base[n] + (dy * a.sp.Wp + dx) * 4;
                        float4 q = make_float4(none, none, none, none);
                        if (two) q = *reinterpret_cast<const float4*>(p + a.x_plane);
                        take(*reinterpret_cast<const float4*>(p), q);
                    }
            }
            if (!real[n] || !two) {
#pragma unroll
                for (int k = 0; k < 8; ++k) if (!real[n] || c0 + k >= a.C) v[k] = 0.f;
            }
            f2 pv[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (AFFINE && K == 2) { v[2 * k] *= 0.25f; v[2 * k + 1] *= 0.25f; }
                big = max3_abs(big, v[2 * k], v[2 * k + 1]);
                pv[k] = f2_of(v[2 * k], v[2 * k + 1]);
            }
            if (a.y) {
                uint4 hi, lo;
                split8(pv, s, hi, lo);
                char* p = yg + (long long)g * 16;
                *reinterpret_cast<uint4*>(p) = hi;
                *reinterpret_cast<uint4*>(p + a.y_plane) = lo;
            }
            if (a.yf && real[n]) {
                float* p = fg + (long long)g * 4;
                *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(pv[0], pv[1]);
                if (two) *reinterpret_cast<ulonglong2*>(p + a.yf_plane) = make_ulonglong2(pv[2], pv[3]);
            }
        }
    }
    const unsigned int most = __reduce_max_sync(0xffffffffu, __float_as_uint(big));
    if ((threadIdx.x & 31) == 0 && most) atomicMax(&word, most);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (word) atomicMax(reinterpret_cast<unsigned int*>(a.y_max), word);
        if (a.y_scale && blockIdx.x == 0 && cg == 0) *a.y_scale = s;
    }
}

constexpr int HEAD_THREADS = 256;

struct HeadArgs {
    const float* x; long long x_plane; Space sp;       // fp32 planes
    int HW;                                            // ... or an NCHW tensor of this many pixels
    int B, C, N;
    const float* scale; const float* shift;            // BatchNorm + ReLU before the average, or nullptr
    float* g;                                          // [B][C] averages
    const float* w; const float* bias;                 // [N][C], [N]
    float* y;                                          // [B][N]
    int vec;                                           // C is a multiple of 4 and w is 16-byte aligned
};

// Global average: one warp per image and 16 channels, so that a 7x7 image's loads (two per lane and four channels) are all in
// flight at once; the 16 sums are added across the lanes by halving both (16 shuffles).  2048 channels, 64 images: 16.3 ->
// 10.8 us against one warp per four channels.
__global__ void __launch_bounds__(HEAD_THREADS) gap_kernel(const HeadArgs a) {
    pdl_enter();
    const int lane = threadIdx.x & 31, c4n = (a.C + 3) / 4, parts = (c4n + 3) / 4;
    for (int wi = (int)(blockIdx.x * (HEAD_THREADS / 32) + (threadIdx.x >> 5)); wi < a.B * parts; wi += (int)gridDim.x * (HEAD_THREADS / 32)) {
        const int b = wi / parts, c4 = (wi - b * parts) * 4;
        const float* p = a.x + (long long)c4 * a.x_plane + (long long)b * a.sp.Lp * 4;
        float sc[16], sh[16], v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const bool has = a.scale && c4 * 4 + k < a.C;
            sc[k] = has ? __ldg(a.scale + c4 * 4 + k) : 0.f; sh[k] = has ? __ldg(a.shift + c4 * 4 + k) : 0.f;
            v[k] = 0.f;
        }
        const int n = a.sp.H * a.sp.W;
#pragma unroll 2
        for (int i = lane; i < n; i += 32) {
            const int yy = i / a.sp.W, xx = i - yy * a.sp.W;
            const float* q = p + ((long long)yy * a.sp.Wp + xx) * 4;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c4 + u < c4n) t = *reinterpret_cast<const float4*>(q + u * a.x_plane);
                if (a.scale) {
                    t.x = max_nan(fmaf(t.x, sc[4 * u], sh[4 * u]), 0.f); t.y = max_nan(fmaf(t.y, sc[4 * u + 1], sh[4 * u + 1]), 0.f);
                    t.z = max_nan(fmaf(t.z, sc[4 * u + 2], sh[4 * u + 2]), 0.f); t.w = max_nan(fmaf(t.w, sc[4 * u + 3], sh[4 * u + 3]), 0.f);
                }
                v[4 * u] += t.x; v[4 * u + 1] += t.y; v[4 * u + 2] += t.z; v[4 * u + 3] += t.w;
            }
        }
        int c = c4 * 4;
#pragma unroll
        for (int d = 16; d >= 2; d >>= 1) {
            const bool upper = lane & d;
#pragma unroll
            for (int k = 0; k < d / 2; ++k) {
                const float keep = upper ? v[k + d / 2] : v[k], send = upper ? v[k] : v[k + d / 2];
                v[k] = keep + __shfl_xor_sync(0xffffffffu, send, d);
            }
            c += upper ? d / 2 : 0;
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        if (!(lane & 1) && c < a.C) a.g[(long long)b * a.C + c] = v[0] / (float)n;
    }
}

// ... of an NCHW tensor: one warp per image and channel.
__global__ void __launch_bounds__(HEAD_THREADS) gap_nchw_kernel(const HeadArgs a) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    for (long long wi = (long long)blockIdx.x * (HEAD_THREADS / 32) + (threadIdx.x >> 5); wi < (long long)a.B * a.C; wi += (long long)gridDim.x * (HEAD_THREADS / 32)) {
        const float* p = a.x + wi * a.HW;
        const int c = (int)(wi % a.C);
        const float sc = a.scale ? __ldg(a.scale + c) : 1.f, sh = a.scale ? __ldg(a.shift + c) : 0.f;
        float s = 0.f;
        for (int i = lane; i < a.HW; i += 32) { const float t = p[i]; s += a.scale ? max_nan(fmaf(t, sc, sh), 0.f) : t; }
        for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane == 0) a.g[wi] = s / (float)a.HW;
    }
}

// Classifier on a few images: one warp per output and up to 4 images, the averages read from cache, the filter row once.
template <int IB>
__global__ void __launch_bounds__(HEAD_THREADS) fc_rows_kernel(const HeadArgs a) {
    pdl_enter();
    const int lane = threadIdx.x & 31, n = (int)(blockIdx.x * (HEAD_THREADS / 32) + (threadIdx.x >> 5)), b0 = (int)blockIdx.y * IB;
    if (n >= a.N) return;
    float s[IB];
#pragma unroll
    for (int i = 0; i < IB; ++i) s[i] = 0.f;
    const float* w = a.w + (long long)n * a.C;
    if (a.vec) {
#pragma unroll 4
        for (int c = lane * 4; c < a.C; c += 128) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(w + c));
#pragma unroll
            for (int i = 0; i < IB; ++i)
                if (b0 + i < a.B) {
                    const float4 g = *reinterpret_cast<const float4*>(a.g + (long long)(b0 + i) * a.C + c);
                    s[i] = fmaf(g.w, t.w, fmaf(g.z, t.z, fmaf(g.y, t.y, fmaf(g.x, t.x, s[i]))));
                }
        }
    } else {
        for (int c = lane; c < a.C; c += 32) {
            const float t = __ldg(w + c);
#pragma unroll
            for (int i = 0; i < IB; ++i) if (b0 + i < a.B) s[i] = fmaf(a.g[(long long)(b0 + i) * a.C + c], t, s[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < IB; ++i) {
        for (int d = 16; d; d >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], d);
        if (lane == 0 && b0 + i < a.B) a.y[(long long)(b0 + i) * a.N + n] = s[i] + (a.bias ? __ldg(a.bias + n) : 0.f);
    }
}

// ... and on many: 16 images x 32 outputs per block.  Both operands pass through shared memory in four stages of 128 channels
// (rows 16 bytes apart in the banks, so that the eight rows a load of a warp touches do not meet), and the channels of a stage
// are dealt to the eight warps, 4 x 4 outputs per lane; their partial sums are added in order.  Reading the operands straight
// from cache the kernel was a chain of L2 round trips: 2048 -> 1000, 64 images, 62 -> 24 us; 512 -> 1000, 256 images, 42 -> 15.
constexpr int FC_B = 16, FC_N = 32, FC_K = 128, FC_ROW = FC_K + 4, FC_STAGES = 4;
constexpr size_t FC_SMEM = sizeof(float) * FC_STAGES * (FC_B + FC_N) * FC_ROW;
static_assert(8 * FC_B * FC_N <= FC_STAGES * (FC_B + FC_N) * FC_ROW, "the partial sums take the stages' place");

template <bool VEC>
__global__ void __launch_bounds__(HEAD_THREADS) fc_tile_kernel(const HeadArgs a) {
    extern __shared__ __align__(16) float fc_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tb = lane & 3, tn = lane >> 2;
    const int n0 = (int)blockIdx.x * FC_N, b0 = (int)blockIdx.y * FC_B, chunks = (a.C + FC_K - 1) / FC_K;
    // rows [first, last) of a stage: the images, then the outputs; what lies behind the last channel is zero
    auto stage = [&](int chunk, int first, int last) {
        if (chunk >= chunks) return;
        float* S = fc_smem + (chunk % FC_STAGES) * (FC_B + FC_N) * FC_ROW;
        constexpr int PER = VEC ? FC_K / 4 : FC_K;
#pragma unroll 6
        for (int i = threadIdx.x; i < (last - first) * PER; i += HEAD_THREADS) {
            const int row = first + i / PER, k = (i % PER) * (VEC ? 4 : 1), c = chunk * FC_K + k;
            const float* src = row < FC_B ? a.g + (long long)min(b0 + row, a.B - 1) * a.C : a.w + (long long)min(n0 + row - FC_B, a.N - 1) * a.C;
            const bool in = c < a.C;
            const uint32_t dst = smem_u32(S + row * FC_ROW + k);
            if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src + (in ? c : 0)), "r"(in ? 16 : 0) : "memory");
            else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src + (in ? c : 0)), "r"(in ? 4 : 0) : "memory");
        }
    };
    // the filter is no earlier launch's output: its first stages are on their way before those end
    for (int k = 0; k < FC_STAGES - 1; ++k) stage(k, FC_B, FC_B + FC_N);
    pdl_enter();
    for (int k = 0; k < FC_STAGES - 1; ++k) {
        stage(k, 0, FC_B);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
    for (int chunk = 0; chunk < chunks; ++chunk) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FC_STAGES - 2) : "memory");
        __syncthreads();
        stage(chunk + FC_STAGES - 1, 0, FC_B + FC_N);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* S = fc_smem + (chunk % FC_STAGES) * (FC_B + FC_N) * FC_ROW + warp * (FC_K / 8);
#pragma unroll
        for (int k = 0; k < FC_K / 8; k += 4) {
            float4 g[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                g[i] = *reinterpret_cast<const float4*>(S + (tb + 4 * i) * FC_ROW + k);
                w[i] = *reinterpret_cast<const float4*>(S + (FC_B + tn + 8 * i) * FC_ROW + k);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    s[i][j] = fmaf(g[i].w, w[j].w, fmaf(g[i].z, w[j].z, fmaf(g[i].y, w[j].y, fmaf(g[i].x, w[j].x, s[i][j]))));
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) fc_smem[warp * FC_B * FC_N + (tb + 4 * i) * FC_N + tn + 8 * j] = s[i][j];
    __syncthreads();
    for (int o = threadIdx.x; o < FC_B * FC_N; o += HEAD_THREADS) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += fc_smem[w * FC_B * FC_N + o];
        const int b = b0 + o / FC_N, n = n0 + o % FC_N;
        if (b < a.B && n < a.N) a.y[(long long)b * a.N + n] = t + (a.bias ? __ldg(a.bias + n) : 0.f);
    }
}

// Inference BatchNorm as scale and shift, in double and rounded once, and {max |scale|, max |shift|}.
__global__ void __launch_bounds__(256) fold_bn_kernel(const float* var, const float* mean, const float* weight, const float* bias, double eps, int n,
                                                      float* scale, float* shift, float* bound) {
    __shared__ unsigned int word;
    unsigned int ms = 0, mt = 0;
    for (int i = threadIdx.x; i < n; i += 256) {
        const double s = (weight ? (double)weight[i] : 1.0) / sqrt((double)var[i] + eps);
        const float fs = (float)s, ft = (float)((bias ? (double)bias[i] : 0.0) - (double)mean[i] * s);
        scale[i] = fs; shift[i] = ft;
        ms = max(ms, __float_as_uint(fs) & 0x7fffffffu); mt = max(mt, __float_as_uint(ft) & 0x7fffffffu);
    }
    ms = block_max(ms, &word);
    mt = block_max(mt, &word);
    if (threadIdx.x == 0) { bound[0] = __uint_as_float(ms); bound[1] = __uint_as_float(mt); }
}

// ---- filters -----------------------------------------------------------------------------------------------------------
struct FilterArgs {
    const float* w; int K, C, R;                       // [K][C][R][R]
    int mode, nt, cblocks;                             // cblocks: channel blocks of 16 (per parity in MODE_S2)
    const float* scale; const float* bias;
    float* stat;                                       // [2 K] scratch: max |w|, sum |w| x |scale| of every output channel
    char* wt; float* meta;
};

// One block per output channel: its largest magnitude and its L1 norm.
__global__ void __launch_bounds__(128) filter_stat_kernel(const FilterArgs a) {
    __shared__ float red[2][4];
    const int k = (int)blockIdx.x, n = a.C * a.R * a.R;
    const float* w = a.w + (long long)k * n;
    float m = 0.f, l = 0.f;
    for (int i = threadIdx.x; i < n; i += 128) { const float t = fabsf(__ldg(w + i)); m = fmaxf(m, t); l += t; }
    for (int d = 16; d; d >>= 1) { m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d)); l += __shfl_xor_sync(0xffffffffu, l, d); }
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = m; red[1][threadIdx.x >> 5] = l; }
    __syncthreads();
    if (threadIdx.x == 0) {
        a.stat[k] = fmaxf(fmaxf(red[0][0], red[0][1]), fmaxf(red[0][2], red[0][3]));
        a.stat[a.K + k] = (red[1][0] + red[1][1] + red[1][2] + red[1][3]) * (a.scale ? fabsf(a.scale[k]) : 1.f);
    }
}

// Filter -> the shared-memory image of every (output block, channel block): [tap][2 words][hi | lo x nt rows][8 halves].
__global__ void __launch_bounds__(256) filter_prepare_kernel(const FilterArgs a) {
    __shared__ unsigned int word;
    unsigned int m = 0, l = 0, bm = 0;
    for (int k = threadIdx.x; k < a.K; k += 256) {
        m = max(m, __float_as_uint(a.stat[k]));
        l = max(l, __float_as_uint(a.stat[a.K + k]));
        if (a.bias) bm = max(bm, __float_as_uint(a.bias[k]) & 0x7fffffffu);
    }
    const float ws = range_scale(__uint_as_float(block_max(m, &word)));
    const float l1 = __uint_as_float(block_max(l, &word)), bmax = __uint_as_float(block_max(bm, &word));
    if (blockIdx.x == 0 && threadIdx.x == 0) { a.meta[0] = ws; a.meta[1] = l1; a.meta[2] = bmax; a.meta[3] = 0.f; }
    const int RR = a.R * a.R, nt = a.nt;
    const int taps_all = a.mode == MODE_S2 ? 9 : a.mode;
    const int n_ocb = (a.K + nt - 1) / nt;
    const long long words = (long long)n_ocb * a.cblocks * taps_all * 4 * nt;      // 16-byte words
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < words; i += (long long)gridDim.x * 256) {
        long long t = i;
        const int nn = (int)(t % nt); t /= nt;
        const int part = (int)(t & 1); t >>= 1;
        const int wd = (int)(t & 1); t >>= 1;
        int tap, cb, parity = 0;
        const long long per_ocb = (long long)a.cblocks * taps_all;
        const int ocb = (int)(t / per_ocb);
        int r = (int)(t - ocb * per_ocb);
        if (a.mode == MODE_S2) {
            // parities in order, each [channel block][tap] with 1, 2, 2, 4 taps
            int before = 0;
            for (parity = 0; parity < 3; ++parity) {
                const int n = taps_of<MODE_S2>(parity) * a.cblocks;
                if (r < before + n) break;
                before += n;
            }
            r -= before;
            const int tp = taps_of<MODE_S2>(parity);
            cb = r / tp; tap = r - cb * tp;
        } else { cb = r / taps_all; tap = r - cb * taps_all; }
        const int oc = ocb * nt + nn;
        uint32_t out[4];
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
            __half h[2];
#pragma unroll
            for (int e1 = 0; e1 < 2; ++e1) {
                const int ch = cb * 16 + wd * 8 + e2 * 2 + e1;
                int c = ch, dy = 0, dx = 0;
                bool ok = oc < a.K;
                if (a.mode == MODE_3x3) { dy = tap / 3; dx = tap % 3; }
                else if (a.mode == MODE_ROW3) { c = ch / 3; dx = ch % 3; dy = tap; }
                else if (a.mode == MODE_S2) {
                    const int pc = 1 + (parity & 1), ti = tap / pc, tj = tap - ti * pc;
                    dy = (parity >> 1) ? 2 * ti : 1; dx = (parity & 1) ? 2 * tj : 1;
                } else if (a.mode == MODE_4x4) {
                    c = ch >> 2;
                    dy = 2 * (tap >> 2) + ((ch >> 1) & 1) - 1; dx = 2 * (tap & 3) + (ch & 1) - 1;
                    ok = ok && dy >= 0 && dy < 7 && dx >= 0 && dx < 7;
                }
                ok = ok && c < a.C;
                float v = ok ? __ldg(a.w + ((long long)oc * a.C + c) * RR + dy * a.R + dx) * ws : 0.f;
                const __half hi = __float2half_rn(v);
                h[e1] = part == 0 ? hi : __float2half_rn((v - __half2float(hi)) * 2048.f);
            }
            const __half2 hh = __halves2half2(h[0], h[1]);
            out[e2] = *reinterpret_cast<const uint32_t*>(&hh);
        }
        *reinterpret_cast<uint4*>(a.wt + i * 16) = make_uint4(out[0], out[1], out[2], out[3]);
    }
}

}  // namespace tdc_pk
