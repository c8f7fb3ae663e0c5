// A chain of convolutions as one object: built once per input shape, then run with one call.
//
// The reference's end-to-end skeletons are C++ programs whose forward is a few hundred bare launches
// (A100-evaluation/EndToEnd/resnet18-tk/src/main.cu:127-155); here a network is a list of prepared launches on packed
// activations (pk.h).  Building it lays out one arena for all intermediates (a buffer is reused when its last reader has
// run), picks the kernel instance of every convolution and fills the argument blocks; running it patches the caller's
// pointers in and issues the launches, about 2 us of host time each, chained by programmatic dependent launch.
#include <cuda_runtime.h>
#include <algorithm>
#include <functional>
#include <map>
#include <mutex>
#include <set>
#include <vector>
#include "../../include/tdc_b200.h"
#include "conv_pk_plan.h"
#include "errors.h"
#include "pk_ops.cuh"

using tdc::fail;
using namespace tdc_pk;

int* tdc_tc_status_word();      // conv_tc.cu: the device status word of the tensor-core kernels

namespace {

std::mutex g_mu;
std::map<int, Facts> g_facts;
std::set<std::pair<int, const void*>> g_opted;

int facts_of_device(Facts* out) {
    int dev;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(TDC_ERR_NO_DEVICE, "cudaGetDevice: %s", cudaGetErrorString(e));
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_facts.find(dev);
    if (it == g_facts.end()) {
        Facts f;
        if ((e = cudaDeviceGetAttribute(&f.smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
            return fail(TDC_ERR_CUDA, "device query: %s", cudaGetErrorString(e));
        f.status = tdc_tc_status_word();
        if (!f.status) return fail(TDC_ERR_CUDA, "the status word has no address");
        it = g_facts.emplace(dev, f).first;
    }
    *out = it->second;
    return TDC_OK;
}

// Opens the whole shared memory of an SM to a kernel, once per device.
int opt_in(const void* fn, int smem_max) {
    int dev;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_opted.insert({dev, fn}).second) return TDC_OK;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
    return e == cudaSuccess ? TDC_OK : fail(TDC_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
}

// A tdc_status; the steps that call other entry points return theirs.
int launch_args(const void* fn, dim3 grid, int threads, int cluster, size_t smem, void** argv, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, argv);
    return e == cudaSuccess ? TDC_OK : fail(TDC_ERR_CUDA, "launch: %s", cudaGetErrorString(e));
}
int launch(const void* fn, dim3 grid, int threads, int cluster, size_t smem, void* args, cudaStream_t st) {
    void* argv[] = {args};
    return launch_args(fn, grid, threads, cluster, smem, argv, st);
}

struct Buffer { size_t bytes = 0, off = 0; int def = -1, last = -1; };

struct Tensor {
    Space s{};
    int C = 0, groups = 0;             // groups of 8 channels in packed form (an even number)
    int pk = -1, f4 = -1;              // buffers, or -1
    int nchw = -1, H = 0, W = 0;       // buffer of an NCHW tensor, and its image
    int range = -1;                    // buffer of the partial maxima a convolution with fp16 parts left of it, or -1
    size_t meta = 0;                   // floats from the start of the meta area
    int slots = 0;                     // partial maxima written so far
};

struct RunArgs {
    char* arena; const float* x; const float* x_absmax; float* y; float* y_absmax; cudaStream_t st;
    bool factors; const float* scale; const float* bias;      // factors: these in place of what the convolution that writes y was built with
};

}  // namespace

struct tdc_net {
    Facts f;
    int device = 0;
    int B = 0, C = 0, H = 0, W = 0;    // the NCHW input
    std::vector<Tensor> tensors;
    std::vector<Buffer> buffers;
    std::vector<std::function<int(const RunArgs&)>> ops;
    size_t meta_floats = 0, meta_off = 0, arena_bytes = 0;
    bool finished = false, packed_y = false;        // packed_y: a convolution on packed activations writes y

    int buffer(size_t bytes) {
        Buffer b;
        b.bytes = (bytes + 255) & ~(size_t)255;
        b.def = b.last = (int)ops.size();
        buffers.push_back(b);
        return (int)buffers.size() - 1;
    }
    void use(int buf) { if (buf >= 0) buffers[buf].last = std::max(buffers[buf].last, (int)ops.size()); }
    int tensor(const Space& s, int C, bool pk, bool f4, int meta_words = META_FLOATS) {
        Tensor t;
        t.s = s; t.C = C; t.groups = ((C + 15) / 16) * 2;
        if (pk) t.pk = buffer((size_t)t.groups * 2 * space_alloc(s) * 16);
        if (f4) t.f4 = buffer((size_t)((C + 3) / 4) * space_alloc(s) * 16);
        t.meta = meta_floats;
        meta_floats += (size_t)meta_words;
        tensors.push_back(t);
        return (int)tensors.size() - 1;
    }
    char* pk_at(const RunArgs& r, const Tensor& t) const { return r.arena + buffers[t.pk].off + (size_t)space_front(t.s) * 16; }
    float* f4_at(const RunArgs& r, const Tensor& t, int c0 = 0) const {
        return reinterpret_cast<float*>(r.arena + buffers[t.f4].off) + (size_t)(c0 / 4) * space_alloc(t.s) * 4 + (size_t)space_front(t.s) * 4;
    }
    float* meta_at(const RunArgs& r, const Tensor& t) const { return reinterpret_cast<float*>(r.arena + meta_off) + t.meta; }
    int nchw_tensor(int C, int H, int W) {
        Tensor t;
        t.C = C; t.H = H; t.W = W;
        t.nchw = buffer(sizeof(float) * (size_t)B * C * H * W);
        tensors.push_back(t);
        return (int)tensors.size() - 1;
    }
    // an NCHW tensor's data; -1: the run's input
    const float* nchw_at(const RunArgs& r, int id) const { return id < 0 ? r.x : reinterpret_cast<const float*>(r.arena + buffers[tensors[id].nchw].off); }
    float* range_at(const RunArgs& r, int id) const { return id < 0 || tensors[id].range < 0 ? nullptr : reinterpret_cast<float*>(r.arena + buffers[tensors[id].range].off); }
    bool is_nchw(int id) const { return id == -1 || (has(id) && tensors[id].nchw >= 0); }
    void use_nchw(int id) { if (id >= 0) { use(tensors[id].nchw); use(tensors[id].range); } }
    static long long pk_plane(const Tensor& t) { return space_alloc(t.s) * 16; }
    static long long f4_plane(const Tensor& t) { return space_alloc(t.s) * 4; }
    bool has(int id) const { return id >= 0 && id < (int)tensors.size(); }
};

namespace {

// Makes a net's device current for as long as it lives: kernels are opened to all of shared memory per device, and a launch on the
// default stream goes to the current one.
struct OnDevice {
    int before = -1;
    explicit OnDevice(int device) {
        int now = -1;
        if (cudaGetDevice(&now) == cudaSuccess && now != device && cudaSetDevice(device) == cudaSuccess) before = now;
    }
    ~OnDevice() { if (before >= 0) cudaSetDevice(before); }
    OnDevice(const OnDevice&) = delete;
};

// Spaces count positions in 32 bits (Space::Lp, the fast divisions): `pad` zeros per row and image included.
bool image_fits(long long B, long long H, long long W) { return (H + 2) * (W + 2) < (1ll << 30) && B * (H + 2) * (W + 2) < (1ll << 31); }

unsigned blocks_for(long long items, const Facts& f) {
    long long b = (items + OPS_THREADS - 1) / OPS_THREADS;
    const long long cap = 2ll * f.sms < PACK_SLOTS ? 2ll * f.sms : PACK_SLOTS;     // what is resident: every further block samples the range again
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

int mode_of(int kind) {
    switch (kind) {
        case TDC_NET_CONV1x1: case TDC_NET_CONV1x1_S2: return MODE_1x1;
        case TDC_NET_CONV3x3: return MODE_3x3;
        case TDC_NET_CONV3x3_S2: return MODE_S2;
        case TDC_NET_CONV7x7_S2: return MODE_4x4;
        case TDC_NET_CONV3x3_ROWS: return MODE_ROW3;
        default: return 0;
    }
}
int filter_channels(int kind, int C) { return kind == TDC_NET_CONV7x7_S2 ? 4 * C : (kind == TDC_NET_CONV3x3_ROWS ? 3 * C : C); }
int filter_size(int kind) { return kind == TDC_NET_CONV7x7_S2 ? 7 : (kind == TDC_NET_CONV1x1 || kind == TDC_NET_CONV1x1_S2 ? 1 : 3); }

// The part of the argument block that follows from the layer: input space, channel blocks, outputs asked for (as flags).
int describe(const Tensor& t, const tdc_net_conv* d, Args* a, int* mode) {
    *mode = mode_of(d->kind);
    if (!*mode) return fail(TDC_ERR_UNSUPPORTED, "convolution kind %d", d->kind);
    if (d->K <= 0) return fail(TDC_ERR_SHAPE, "K=%d", d->K);
    *a = Args{};
    a->sp = t.s;
    if (d->kind == TDC_NET_CONV3x3_S2 || d->kind == TDC_NET_CONV1x1_S2) {
        if (!t.s.split_B) return fail(TDC_ERR_UNSUPPORTED, "a stride-2 convolution reads a tensor split by parity");
        a->sp = make_space(t.s.split_B, t.s.H, t.s.W, t.s.pad);      // the outputs: one sub-image of every image
    } else if (t.s.split_B && d->kind != TDC_NET_CONV1x1) return fail(TDC_ERR_UNSUPPORTED, "this convolution cannot read a tensor split by parity");
    if (d->kind == TDC_NET_CONV7x7_S2 && t.s.pad < 2) return fail(TDC_ERR_UNSUPPORTED, "the 7x7 form reads an input packed for it");
    a->cbl = t.groups / 2;
    a->nkb = *mode == MODE_S2 ? 4 * a->cbl : a->cbl;
    a->K = d->K;
    a->k16 = (d->K + 15) & ~15;
    a->pool = d->pool;
    if (d->pool) {
        if ((d->pool != POOL_2x2 && d->pool != POOL_3x3) || !d->relu || d->residual >= 0 || d->out_split || (d->out & TDC_NET_NCHW) || a->sp.H < 2 || a->sp.W < 2)
            return fail(TDC_ERR_UNSUPPORTED, "pooling goes with ReLU, without a residual, into the net");
    }
    // only whether they are there matters for the choice of a kernel
    static char here;
    if (d->out & TDC_NET_PACKED) a->y = &here;
    if (d->out & TDC_NET_PLANES) a->yf = reinterpret_cast<float*>(&here);
    if (d->out & TDC_NET_NCHW) a->nchw = reinterpret_cast<float*>(&here);
    if (d->residual >= 0) a->res = reinterpret_cast<const float*>(&here);
    return TDC_OK;
}

int describe(const tdc_net* n, int src, const tdc_net_conv* d, Args* a, int* mode) {
    if (!n->has(src) || n->tensors[src].pk < 0) return fail(TDC_ERR_UNSUPPORTED, "tensor %d has no packed form", src);
    return describe(n->tensors[src], d, a, mode);
}

// Picks the instance (or checks the one named) and fills in what tdc_net_conv_plan promises.
int plan(const Tensor& t, const Facts& f, tdc_net_conv* d) {
    Args a;
    int mode;
    const int rc = describe(t, d, &a, &mode);
    if (rc) return rc;
    Choice c{d->nt, d->mt, d->ks};
    Launch l;
    if (!d->nt) {
        if (!choose(a, mode, f, &c)) return fail(TDC_ERR_SMEM, "no kernel on packed activations fits this convolution");
    } else if ((c.nt != 32 && c.nt != 64 && c.nt != 128) || (!c.ks && c.mt != 1 && c.mt != 2))
        return fail(TDC_ERR_UNSUPPORTED, "nt=%d mt=%d ks=%d", c.nt, c.mt, c.ks);
    double clocks = 0.0;
    if (!configure(a, mode, c, f, &l, &clocks)) return fail(TDC_ERR_SMEM, "nt=%d mt=%d ks=%d does not fit this convolution", c.nt, c.mt, c.ks);
    // memory: from HBM where the launch moves more than L2 holds, else out of L2 (bytes per clock of the whole chip)
    const double out = (a.y ? 4.0 : 0.0) + (a.yf ? 4.0 : 0.0) + (a.nchw ? 4.0 : 0.0) + (a.res ? 4.0 : 0.0);
    const double bytes = (double)t.groups * 32.0 * (double)t.s.total + out * d->K * (double)a.sp.total / (d->pool ? 4.0 : 1.0);
    const double mem = 4000.0 + bytes / (bytes > 80e6 ? 2600.0 : 6500.0);
    d->nt = c.nt; d->mt = c.mt; d->ks = c.ks; d->clocks = (float)(clocks > mem ? clocks : mem);
    d->filter_bytes = tdc_net_filter_bytes(d->kind, d->K, t.C, c.nt);
    return TDC_OK;
}

}  // namespace

extern "C" {

int tdc_net_create(tdc_net** out, int B, int C, int H, int W) {
    if (!out) return fail(TDC_ERR_NULL, "out is NULL");
    if (B <= 0 || C <= 0 || H <= 0 || W <= 0 || !image_fits(B, H, W)) return fail(TDC_ERR_SHAPE, "B=%d C=%d H=%d W=%d", B, C, H, W);
    Facts f;
    const int rc = facts_of_device(&f);
    if (rc) return rc;
    tdc_net* n = new tdc_net;
    n->f = f; n->B = B; n->C = C; n->H = H; n->W = W;
    cudaGetDevice(&n->device);
    *out = n;
    return TDC_OK;
}

void tdc_net_destroy(tdc_net* n) { delete n; }

int tdc_net_pack(tdc_net* n, int kind, int* out) {
    if (!n || !out) return fail(TDC_ERR_NULL, "net and out must be non-NULL");
    const bool want_exact = kind & TDC_NET_PACK_EXACT;
    kind &= ~TDC_NET_PACK_EXACT;
    if (kind < PACK_SAME || kind > PACK_ROW3) return fail(TDC_ERR_UNSUPPORTED, "pack kind %d", kind);
    if (!n->tensors.empty()) return fail(TDC_ERR_UNSUPPORTED, "packing the input is a net's first step");
    Space s;
    int C = n->C;
    if (kind == PACK_S2D) { s = make_space(n->B, (n->H + 1) / 2, (n->W + 1) / 2, 2); C *= 4; }
    else { s = make_space(n->B, n->H, n->W, 1, kind == PACK_SPLIT); if (kind == PACK_ROW3) C *= 3; }
    const long long items = (space_front(s) + s.total) * (long long)(((C + 15) / 16) * 2);   // (also bounds H * W)
    if (items >= (1ll << 31) || s.total >= (1ll << 30)) return fail(TDC_ERR_SHAPE, "input too large for the packed form");
    const int id = n->tensor(s, C, true, false, 1 + PACK_SLOTS);
    Tensor& t = n->tensors[id];
    PackArgs a{};
    a.B = n->B; a.C = n->C; a.H = n->H; a.W = n->W;
    a.groups = t.groups; a.front = space_front(s); a.d = s; a.y_plane = tdc_net::pk_plane(t); a.status = n->f.status;
    const long long values = (long long)n->B * n->C * n->H * n->W;
    const bool exact = values <= PACK_EXACT;
    a.sample_step = (uint32_t)((values + 3 * OPS_THREADS - 1) / (3 * OPS_THREADS));
    unsigned grid = blocks_for(items, n->f);
    if (exact) grid = std::min<unsigned>((grid + PACK_CLUSTER - 1) / PACK_CLUSTER, PACK_SLOTS / PACK_CLUSTER) * PACK_CLUSTER;
    t.slots = (int)grid;
    const void* const forms[2][4] = {{(const void*)&pack_kernel<PACK_SAME, false>, (const void*)&pack_kernel<PACK_SPLIT, false>, (const void*)&pack_kernel<PACK_S2D, false>, (const void*)&pack_kernel<PACK_ROW3, false>},
                                     {(const void*)&pack_kernel<PACK_SAME, true>, (const void*)&pack_kernel<PACK_SPLIT, true>, (const void*)&pack_kernel<PACK_S2D, true>, (const void*)&pack_kernel<PACK_ROW3, true>}};
    const void* fn = forms[exact][kind];
    const int range = want_exact && !exact ? n->buffer(sizeof(float) * tdc_tc::ABSMAX_SLOTS) : -1;
    if (range >= 0) {
        const unsigned blocks = (unsigned)std::min<long long>((values / 4 + OPS_THREADS - 1) / OPS_THREADS, 2ll * n->f.sms < tdc_tc::ABSMAX_SLOTS ? 2ll * n->f.sms : tdc_tc::ABSMAX_SLOTS);
        n->ops.push_back([n, range, values, blocks](const RunArgs& r) {
            if (r.x_absmax) return (int)TDC_OK;
            const float* x = r.x;
            float* slots = reinterpret_cast<float*>(r.arena + n->buffers[range].off);
            long long count = values;
            int n_slots = tdc_tc::ABSMAX_SLOTS;
            void* argv[] = {&x, &count, &slots, &n_slots};
            return launch_args((const void*)&range_kernel, dim3(blocks), OPS_THREADS, 1, 0, argv, r.st);
        });
        n->use(range);
        n->use(t.pk);
    }
    n->ops.push_back([n, id, a, grid, fn, exact, range](const RunArgs& r) {
        PackArgs p = a;
        const Tensor& t = n->tensors[id];
        p.x = r.x; p.absmax = r.x_absmax || range < 0 ? r.x_absmax : reinterpret_cast<const float*>(r.arena + n->buffers[range].off); p.absmax_n = tdc_tc::ABSMAX_SLOTS;
        p.y = n->pk_at(r, t);
        p.y_scale = n->meta_at(r, t); p.y_slots = p.y_scale + 1;
        p.zero = p.y_slots + PACK_SLOTS; p.zeros = (int)n->meta_floats - (1 + PACK_SLOTS);
        return launch(fn, dim3(grid), OPS_THREADS, exact ? PACK_CLUSTER : 1, 0, &p, r.st);
    });
    *out = id;
    return TDC_OK;
}

int tdc_net_conv_plan(tdc_net* n, int src, tdc_net_conv* d) {
    if (!n || !d) return fail(TDC_ERR_NULL, "net and conv must be non-NULL");
    if (!n->has(src) || n->tensors[src].pk < 0) return fail(TDC_ERR_UNSUPPORTED, "tensor %d has no packed form", src);
    return plan(n->tensors[src], n->f, d);
}

int tdc_net_estimate(int B, int C, int H, int W, int split, tdc_net_conv* d) {
    if (!d) return fail(TDC_ERR_NULL, "conv must be non-NULL");
    if (B <= 0 || C <= 0 || H <= 0 || W <= 0 || !image_fits(B, H, W)) return fail(TDC_ERR_SHAPE, "B=%d C=%d H=%d W=%d", B, C, H, W);
    Facts f;
    const int rc = facts_of_device(&f);
    if (rc) return rc;
    Tensor t;
    t.s = make_space(B, H, W, d->kind == TDC_NET_CONV7x7_S2 ? 2 : 1, split != 0); t.C = C; t.groups = ((C + 15) / 16) * 2;
    return plan(t, f, d);
}

int tdc_net_fold_bn(const float* var, const float* mean, const float* weight, const float* bias, double eps, int n, float* scale, float* shift, float* bound, void* stream) {
    if (!var || !mean || !scale || !shift || !bound) return fail(TDC_ERR_NULL, "var, mean, scale, shift and bound must be non-NULL");
    if (n <= 0) return fail(TDC_ERR_SHAPE, "n=%d", n);
    fold_bn_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(var, mean, weight, bias, eps, n, scale, shift, bound);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TDC_OK : fail(TDC_ERR_CUDA, "fold launch: %s", cudaGetErrorString(e));
}

// A prepared filter: the operand blocks, then {scale, bound, largest |bias|} and scratch for the channels' statistics.
size_t tdc_net_filter_bytes(int kind, int K, int C_packed, int nt) {
    const int mode = mode_of(kind);
    return mode && K > 0 && C_packed > 0 && nt > 0 ? filter_bytes(mode, K, C_packed, nt) + 64 + sizeof(float) * 2 * (size_t)K : 0;
}

int tdc_net_filter_prepare(int kind, int K, int C, int nt, const float* w, const float* scale, const float* bias, void* out, void* stream) {
    if (!w || !out) return fail(TDC_ERR_NULL, "w and out must be non-NULL");
    const int mode = mode_of(kind);
    if (!mode || K <= 0 || C <= 0 || (nt != 32 && nt != 64 && nt != 128)) return fail(TDC_ERR_UNSUPPORTED, "kind=%d K=%d C=%d nt=%d", kind, K, C, nt);
    if (reinterpret_cast<uintptr_t>(out) % 16) return fail(TDC_ERR_UNSUPPORTED, "a prepared filter is 16-byte aligned");
    const int Cp = filter_channels(kind, C);
    const size_t bytes = filter_bytes(mode, K, Cp, nt);
    FilterArgs a{};
    a.w = w; a.K = K; a.C = C; a.R = filter_size(kind); a.mode = mode; a.nt = nt; a.cblocks = (Cp + 15) / 16;
    a.scale = scale; a.bias = bias;
    a.wt = static_cast<char*>(out);
    a.meta = reinterpret_cast<float*>(a.wt + bytes);
    a.stat = a.meta + 16;
    filter_stat_kernel<<<(unsigned)K, 128, 0, (cudaStream_t)stream>>>(a);
    const long long words = (long long)(bytes / 16);
    filter_prepare_kernel<<<(unsigned)std::min<long long>((words + 255) / 256, 592), 256, 0, (cudaStream_t)stream>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TDC_OK : fail(TDC_ERR_CUDA, "filter launch: %s", cudaGetErrorString(e));
}

int tdc_net_add_conv(tdc_net* n, int src, const tdc_net_conv* d, int* out) {
    if (!n || !d || !out || !d->filter) return fail(TDC_ERR_NULL, "net, conv, filter and out must be non-NULL");
    if (n->finished) return fail(TDC_ERR_UNSUPPORTED, "the net is finished");
    Args a;
    int mode;
    int rc = describe(n, src, d, &a, &mode);
    if (rc) return rc;
    const OnDevice here(n->device);
    const Choice c{d->nt, d->mt, d->ks};
    Launch l;
    if (!configure(a, mode, c, n->f, &l, nullptr)) return fail(TDC_ERR_SMEM, "nt=%d mt=%d ks=%d does not fit this convolution", c.nt, c.mt, c.ks);
    const void* fn = conv_kernel(c, mode, a.pool);
    if ((rc = opt_in(fn, n->f.smem_max))) return rc;
    const int srcC = n->tensors[src].C;
    a.x_plane = tdc_net::pk_plane(n->tensors[src]);
    a.x_slots = n->tensors[src].slots;
    a.wt = static_cast<const char*>(d->filter);
    a.w_meta = reinterpret_cast<const float*>(a.wt + filter_bytes(mode, d->K, srcC, c.nt));
    a.scale = d->scale; a.bias = d->bias; a.relu = d->relu && !d->pool ? 1 : 0;      // (a pooled maximum starts at zero)
    a.rz_unit = d->unbiased ? 0x1p-26f * (mode == MODE_S2 ? 2.25f : (float)mode) / (float)a.nmain : 0.f;
    a.status = n->f.status;
    n->use(n->tensors[src].pk);
    if (d->residual >= 0) {
        if (!n->has(d->residual) || n->tensors[d->residual].f4 < 0) return fail(TDC_ERR_UNSUPPORTED, "the residual has no fp32 planes");
        const Tensor& t = n->tensors[d->residual];
        if (t.s.total != a.sp.total || t.s.Wp != a.sp.Wp || t.C != d->K || t.s.split_B != a.sp.split_B) return fail(TDC_ERR_SHAPE, "the residual does not match the output");
        a.res_plane = tdc_net::f4_plane(t);
        n->use(t.f4);
    }
    const bool to_net = d->out & (TDC_NET_PACKED | TDC_NET_PLANES);
    if (to_net && (d->out & TDC_NET_NCHW)) return fail(TDC_ERR_UNSUPPORTED, "an output is NCHW or stays in the net");
    const bool ceil = d->pool == POOL_3x3;
    const Space pooled = make_space(a.sp.nimg, (a.sp.H + ceil) / 2, (a.sp.W + ceil) / 2, 1);
    int id = -1, into_c = 0;
    if (to_net) {
        if (d->into >= 0) {                // fp32 planes of a tensor that exists: from channel into_c on
            if (!n->has(d->into) || n->tensors[d->into].f4 < 0 || (d->out & TDC_NET_PACKED)) return fail(TDC_ERR_UNSUPPORTED, "only fp32 planes are written into an existing tensor");
            const Tensor& t = n->tensors[d->into];
            if (d->into_c % 4 || d->into_c + d->K > t.C || d->K % 4) return fail(TDC_ERR_SHAPE, "channels [%d, %d) of %d", d->into_c, d->into_c + d->K, t.C);
            if (d->pool) a.map = MAP_SPACE;
            const Space& o = d->pool ? pooled : a.sp;
            if (t.s.total != o.total || t.s.Wp != o.Wp || t.s.split_B || a.sp.split_B) return fail(TDC_ERR_SHAPE, "the tensor written into has another shape");
            id = d->into; into_c = d->into_c;
            n->use(t.f4);
        } else {
            Space s = a.sp;
            if (d->pool) { s = pooled; a.map = MAP_SPACE; }
            else if (d->out_split) {
                if (a.sp.split_B) return fail(TDC_ERR_UNSUPPORTED, "the output is split already");
                s = make_space(a.sp.nimg, a.sp.Hf, a.sp.Wf, 1, true);
                a.map = MAP_SPLIT;
            } else if (a.sp.pad != 1) { s = make_space(a.sp.nimg, a.sp.H, a.sp.W, 1); a.map = MAP_SPACE; }
            if (s.total >= (1ll << 30)) return fail(TDC_ERR_SHAPE, "output too large");
            id = n->tensor(s, d->K, d->out & TDC_NET_PACKED, d->out & TDC_NET_PLANES);
        }
        Tensor& t = n->tensors[id];
        a.dsp = t.s; a.front = space_front(t.s);
        a.y_plane = tdc_net::pk_plane(t); a.yf_plane = tdc_net::f4_plane(t);
        t.slots = 1;
    }
    const int res = d->residual, flags = d->out;
    const bool fresh = d->into < 0;
    if (id < 0) n->packed_y = true;
    n->ops.push_back([n, src, id, res, flags, into_c, fresh, a, l, fn](const RunArgs& r) {
        Args p = a;
        const Tensor& s = n->tensors[src];
        p.x = n->pk_at(r, s); p.x_meta = n->meta_at(r, s);
        p.res = nullptr; p.y = nullptr; p.yf = nullptr; p.nchw = nullptr;
        if (res >= 0) { p.res = n->f4_at(r, n->tensors[res]); p.res_meta = n->meta_at(r, n->tensors[res]); }
        if (id >= 0) {
            const Tensor& t = n->tensors[id];
            if (flags & TDC_NET_PACKED) p.y = n->pk_at(r, t);
            if (flags & TDC_NET_PLANES) p.yf = n->f4_at(r, t, into_c);
            float* m = n->meta_at(r, t);
            p.y_scale = fresh ? m : nullptr;
            p.y_slots = m + 1;
        } else {
            p.nchw = r.y; p.y_slots = r.y_absmax; p.y_slots_clear = tdc_tc::ABSMAX_SLOTS;
            if (r.factors) { p.scale = r.scale; p.bias = r.bias; }      // (the bounds taken from those it was built with serve packed outputs only)
        }
        return launch(fn, dim3(l.grid), l.threads, l.cluster, l.smem, &p, r.st);
    });
    *out = id;
    return TDC_OK;
}

int tdc_net_planes(tdc_net* n, int B, int C, int H, int W, int* out) {
    if (!n || !out) return fail(TDC_ERR_NULL, "net and out must be non-NULL");
    if (B <= 0 || C <= 0 || H <= 0 || W <= 0 || !image_fits(B, H, W)) return fail(TDC_ERR_SHAPE, "B=%d C=%d H=%d W=%d", B, C, H, W);
    *out = n->tensor(make_space(B, H, W, 1), C, false, true);
    return TDC_OK;
}

int tdc_net_pool(tdc_net* n, int src, const tdc_net_pool_desc* d, int* out) {
    if (!n || !d || !out) return fail(TDC_ERR_NULL, "net, pool and out must be non-NULL");
    if (!n->has(src) || n->tensors[src].f4 < 0 || n->tensors[src].s.split_B) return fail(TDC_ERR_UNSUPPORTED, "pooling reads fp32 planes");
    const Tensor x = n->tensors[src];
    const bool affine = d->scale != nullptr;
    if (affine ? (d->k != 1 && d->k != 2) || d->stride != d->k || d->pad : d->k < 1 || d->stride < 1 || d->pad < 0 || 2 * d->pad > d->k)
        return fail(TDC_ERR_UNSUPPORTED, "window %d stride %d padding %d", d->k, d->stride, d->pad);
    const int C = d->channels ? d->channels : x.C;
    if (C > x.C) return fail(TDC_ERR_SHAPE, "%d of %d channels", C, x.C);
    const int Ho = (x.s.H + 2 * d->pad - d->k) / d->stride + 1, Wo = (x.s.W + 2 * d->pad - d->k) / d->stride + 1;
    if (Ho <= 0 || Wo <= 0) return fail(TDC_ERR_SHAPE, "window larger than the image");
    const Space s = make_space(x.s.nimg, Ho, Wo, 1);
    n->use(x.f4);
    int id;
    const bool fresh = d->into < 0;
    if (fresh) id = n->tensor(s, C, d->out & TDC_NET_PACKED, d->out & TDC_NET_PLANES);
    else {
        if (!n->has(d->into) || n->tensors[d->into].f4 < 0 || d->out != TDC_NET_PLANES) return fail(TDC_ERR_UNSUPPORTED, "only fp32 planes are written into an existing tensor");
        const Tensor& t = n->tensors[d->into];
        if (t.s.total != s.total || t.s.Wp != s.Wp || C > t.C) return fail(TDC_ERR_SHAPE, "the tensor written into has another shape");
        id = d->into;
        n->use(t.f4);
    }
    Tensor& t = n->tensors[id];
    PoolArgs a{};
    a.x_plane = tdc_net::f4_plane(x); a.sp = x.s;
    a.C = C; a.k = d->k; a.stride = d->stride; a.pad = d->pad;
    a.scale = d->scale; a.shift = d->shift; a.bound = d->bound;
    if (affine && (!d->shift || !d->bound)) return fail(TDC_ERR_NULL, "scale comes with shift and bound");
    a.d = s;
    const bool packed = d->out & TDC_NET_PACKED;
    a.front = packed ? space_front(s) : 0;
    const int groups = packed ? ((C + 15) / 16) * 2 : (C + 7) / 8;
    a.y_plane = tdc_net::pk_plane(t); a.yf_plane = tdc_net::f4_plane(t);
    if (s.total + a.front >= (1ll << 30) || groups > 65535) return fail(TDC_ERR_SHAPE, "tensor too large");
    t.slots = 1;
    const void* fn = affine ? (d->k == 2 ? (const void*)&pool_pk_kernel<true, 2> : (const void*)&pool_pk_kernel<true, 1>)
                            : d->k == 3 ? (const void*)&pool_pk_kernel<false, 3> : d->k == 2 ? (const void*)&pool_pk_kernel<false, 2> : (const void*)&pool_pk_kernel<false, 0>;
    // a few rounds of blocks over the chip, none with less than one pass of its threads
    const long long per = (long long)POOL_THREADS * (d->k == 1 ? PoolItems<1>::N : d->k == 2 ? PoolItems<2>::N : 1);
    const long long want = ((long long)n->f.sms * 8 + groups - 1) / groups, most = (s.total + a.front + per - 1) / per;
    const dim3 grid((unsigned)std::max(1ll, std::min(want, most)), (unsigned)groups);
    n->ops.push_back([n, src, id, packed, flags = d->out, fresh, a, grid, fn](const RunArgs& r) {
        PoolArgs p = a;
        const Tensor &x = n->tensors[src], &t = n->tensors[id];
        p.x = n->f4_at(r, x); p.x_max = n->meta_at(r, x) + 1;
        if (packed) p.y = n->pk_at(r, t);
        if (flags & TDC_NET_PLANES) p.yf = n->f4_at(r, t);
        float* m = n->meta_at(r, t);
        p.y_scale = fresh ? m : nullptr; p.y_max = m + 1;
        return launch(fn, grid, POOL_THREADS, 1, 0, &p, r.st);
    });
    *out = id;
    return TDC_OK;
}

// ---- NCHW steps: the layer-by-layer kernels as steps of a net ---------------------------------------------------------------
// (their launches come from the same entry points a caller would use one by one; what a net saves is the host time between them)
static int nchw_dims(const tdc_net* n, int src, int* C, int* H, int* W) {
    if (!n->is_nchw(src)) return fail(TDC_ERR_UNSUPPORTED, "tensor %d is not NCHW", src);
    if (src < 0) { *C = n->C; *H = n->H; *W = n->W; }
    else { *C = n->tensors[src].C; *H = n->tensors[src].H; *W = n->tensors[src].W; }
    return TDC_OK;
}

int tdc_net_nchw_conv(tdc_net* n, int src, const tdc_net_nchw* d, int* out) {
    if (!n || !d || !out || !d->filter) return fail(TDC_ERR_NULL, "net, conv, filter and out must be non-NULL");
    int C, H, W;
    int rc = nchw_dims(n, src, &C, &H, &W);
    if (rc) return rc;
    if (d->K <= 0 || d->R <= 0 || d->S <= 0 || d->stride <= 0 || d->pad < 0 || H + 2 * d->pad < d->R || W + 2 * d->pad < d->S)
        return fail(TDC_ERR_SHAPE, "K=%d filter %dx%d stride %d padding %d on %dx%d", d->K, d->R, d->S, d->stride, d->pad, H, W);
    const int Ho = (H + 2 * d->pad - d->R) / d->stride + 1, Wo = (W + 2 * d->pad - d->S) / d->stride + 1;
    if (d->residual >= 0 && (!n->is_nchw(d->residual) || n->tensors[d->residual].C != d->K || n->tensors[d->residual].H != Ho || n->tensors[d->residual].W != Wo))
        return fail(TDC_ERR_SHAPE, "the residual does not match the output");
    if (d->plan && (d->plan->C != C || d->plan->K != d->K)) return fail(TDC_ERR_SHAPE, "the plan is for another layer");
    n->use_nchw(src);
    n->use_nchw(d->residual);
    const bool tc = d->plan != nullptr, to_y = d->to_y != 0;
    const int id = to_y ? -1 : n->nchw_tensor(d->K, Ho, Wo);
    if (tc && d->plan->mode == 4 && !to_y) n->tensors[id].range = n->buffer(sizeof(float) * tdc_tc::ABSMAX_SLOTS);
    const tdc_net_nchw a = *d;
    const tdc_tc_plan plan = d->plan ? *d->plan : tdc_tc_plan{};
    n->ops.push_back([n, src, id, a, plan, tc, to_y, C, H, W](const RunArgs& r) {
        const tdc_epilogue e{a.scale, a.bias, a.residual >= 0 ? n->nchw_at(r, a.residual) : nullptr, a.relu};
        float* y = to_y ? r.y : const_cast<float*>(n->nchw_at(r, id));
        if (tc && plan.mode == 4)          // (the maxima of one step's output are the range of the next one's input)
            return tdc_conv2d_tc_ranged(&plan, n->nchw_at(r, src), a.filter, y, n->B, H, W, &e, a.flags, src < 0 ? r.x_absmax : n->range_at(r, src),
                                                    to_y ? r.y_absmax : n->range_at(r, id), r.st);
        if (tc) return tdc_conv2d_tc(&plan, n->nchw_at(r, src), a.filter, y, n->B, H, W, &e, a.flags, r.st);
        return tdc_conv2d_epi_f32(n->nchw_at(r, src), static_cast<const float*>(a.filter), y, n->B, C, H, W, a.K, a.R, a.S, a.pad, a.stride,
                                              TDC_W_CRSK, &e, nullptr, r.st);
    });
    *out = id;
    return TDC_OK;
}

int tdc_net_nchw_pool(tdc_net* n, int src, int k, int stride, int pad, int mode, int* out) {
    if (!n || !out) return fail(TDC_ERR_NULL, "net and out must be non-NULL");
    int C, H, W;
    const int rc = nchw_dims(n, src, &C, &H, &W);
    if (rc) return rc;
    if (k <= 0 || stride <= 0 || pad < 0 || H + 2 * pad < k || W + 2 * pad < k) return fail(TDC_ERR_SHAPE, "window %d stride %d padding %d on %dx%d", k, stride, pad, H, W);
    n->use_nchw(src);
    const int id = n->nchw_tensor(C, (H - k + 2 * pad) / stride + 1, (W - k + 2 * pad) / stride + 1);
    n->ops.push_back([n, src, id, C, H, W, k, stride, pad, mode](const RunArgs& r) {
        return tdc_pool2d_f32(n->nchw_at(r, src), const_cast<float*>(n->nchw_at(r, id)), n->B, C, H, W, k, k, pad, stride, mode, r.st);
    });
    *out = id;
    return TDC_OK;
}

int tdc_net_nchw_buffer(tdc_net* n, int C, int H, int W, int* out) {
    if (!n || !out) return fail(TDC_ERR_NULL, "net and out must be non-NULL");
    if (C <= 0 || H <= 0 || W <= 0) return fail(TDC_ERR_SHAPE, "C=%d H=%d W=%d", C, H, W);
    *out = n->nchw_tensor(C, H, W);
    return TDC_OK;
}

int tdc_net_nchw_affine(tdc_net* n, int src, int channels, const float* scale, const float* shift, int relu, int into, int into_c, int* out) {
    if (!n || !out) return fail(TDC_ERR_NULL, "net and out must be non-NULL");
    int C, H, W;
    const int rc = nchw_dims(n, src, &C, &H, &W);
    if (rc) return rc;
    const int c = channels ? channels : C;
    if (c < 0 || c > C) return fail(TDC_ERR_SHAPE, "%d of %d channels", c, C);
    n->use_nchw(src);
    int id = into;
    if (into < 0) id = n->nchw_tensor(c, H, W);
    else {
        if (!n->is_nchw(into) || n->tensors[into].H != H || n->tensors[into].W != W || into_c < 0 || into_c + c > n->tensors[into].C)
            return fail(TDC_ERR_SHAPE, "the tensor written into has another shape");
        n->use_nchw(into);
    }
    const int c0 = into < 0 ? 0 : into_c;
    const long long xs = (long long)C * H * W, ys = (long long)n->tensors[id].C * H * W;
    n->ops.push_back([n, src, id, c, c0, H, W, xs, ys, scale, shift, relu](const RunArgs& r) {
        return tdc_affine_relu_f32(n->nchw_at(r, src), const_cast<float*>(n->nchw_at(r, id)) + (long long)c0 * H * W, scale, shift, n->B, c, H * W, xs, ys, relu, r.st);
    });
    *out = id;
    return TDC_OK;
}

int tdc_net_head(tdc_net* n, int src, const float* scale, const float* shift, const float* w, const float* bias, int N) {
    if (!n) return fail(TDC_ERR_NULL, "net must be non-NULL");
    if (!n->has(src) || (n->tensors[src].nchw < 0 && (n->tensors[src].f4 < 0 || n->tensors[src].s.split_B))) return fail(TDC_ERR_UNSUPPORTED, "the head reads fp32 planes or an NCHW tensor");
    if (w && N <= 0) return fail(TDC_ERR_SHAPE, "N=%d", N);
    const Tensor x = n->tensors[src];
    HeadArgs a{};
    a.B = n->B; a.C = x.C; a.N = N;
    const bool planes = x.nchw < 0;
    if (planes) { a.x_plane = tdc_net::f4_plane(x); a.sp = x.s; }
    else a.HW = x.H * x.W;
    a.scale = scale; a.shift = shift; a.w = w; a.bias = bias;
    a.vec = a.C % 4 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0;
    n->use(planes ? x.f4 : x.nchw);
    const int g = w ? n->buffer(sizeof(float) * (size_t)a.B * a.C) : -1;
    const long long warps = (long long)a.B * (planes ? (a.C + 15) / 16 : a.C);
    const unsigned gap_grid = (unsigned)std::min<long long>((warps + 7) / 8, (long long)n->f.sms * 8);
    n->ops.push_back([n, src, g, a, planes, gap_grid](const RunArgs& r) {
        HeadArgs p = a;
        p.x = planes ? n->f4_at(r, n->tensors[src]) : n->nchw_at(r, src);
        p.g = g < 0 ? r.y : reinterpret_cast<float*>(r.arena + n->buffers[g].off);
        return launch(planes ? (const void*)&gap_kernel : (const void*)&gap_nchw_kernel, dim3(gap_grid), HEAD_THREADS, 1, 0, &p, r.st);
    });
    if (!w) return TDC_OK;
    n->use(g);
    // few images: a warp per output keeps every SM busy reading the filter; many: tiles reuse both operands
    const bool tile = a.B >= 16;
    const void* fc = a.vec ? (const void*)&fc_tile_kernel<true> : (const void*)&fc_tile_kernel<false>;
    if (tile) { const OnDevice here(n->device); const int rc = opt_in(fc, n->f.smem_max); if (rc) return rc; }
    n->ops.push_back([n, g, a, tile, fc](const RunArgs& r) {
        HeadArgs p = a;
        p.g = reinterpret_cast<float*>(r.arena + n->buffers[g].off); p.y = r.y;
        if (tile) return launch(fc, dim3((a.N + FC_N - 1) / FC_N, (a.B + FC_B - 1) / FC_B), HEAD_THREADS, 1, FC_SMEM, &p, r.st);
        if (a.B == 1) return launch((const void*)&fc_rows_kernel<1>, dim3((a.N + 7) / 8, 1), HEAD_THREADS, 1, 0, &p, r.st);
        return launch((const void*)&fc_rows_kernel<4>, dim3((a.N + 7) / 8, (a.B + 3) / 4), HEAD_THREADS, 1, 0, &p, r.st);
    });
    return TDC_OK;
}

int tdc_net_finish(tdc_net* n, size_t* arena_bytes) {
    if (!n || !arena_bytes) return fail(TDC_ERR_NULL, "net and arena_bytes must be non-NULL");
    if (!n->finished) {
        // largest buffers first, each at the lowest offset that is free while it lives
        std::vector<int> order(n->buffers.size());
        for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
        std::sort(order.begin(), order.end(), [&](int p, int q) { return n->buffers[p].bytes > n->buffers[q].bytes; });
        size_t top = 0;
        std::vector<int> placed;
        for (int i : order) {
            Buffer& b = n->buffers[i];
            std::vector<std::pair<size_t, size_t>> busy;
            for (int j : placed) {
                const Buffer& o = n->buffers[j];
                if (o.def <= b.last && b.def <= o.last) busy.push_back({o.off, o.off + o.bytes});
            }
            std::sort(busy.begin(), busy.end());
            size_t at = 0;
            for (const auto& s : busy) {
                if (at + b.bytes <= s.first) break;
                at = std::max(at, s.second);
            }
            b.off = at;
            top = std::max(top, at + b.bytes);
            placed.push_back(i);
        }
        n->meta_off = top;
        n->arena_bytes = top + ((n->meta_floats * sizeof(float) + 255) & ~(size_t)255);
        n->finished = true;
    }
    *arena_bytes = n->arena_bytes;
    return TDC_OK;
}

static int run(const tdc_net* n, RunArgs r, size_t arena_bytes) {
    if (!n || !r.x || !r.y || !r.arena) return fail(TDC_ERR_NULL, "net, x, y and arena must be non-NULL");
    if (!n->finished) return fail(TDC_ERR_UNSUPPORTED, "the net is not finished");
    if (r.factors && !n->packed_y) return fail(TDC_ERR_UNSUPPORTED, "scale and bias per run go to a net that ends in a convolution on packed activations");
    if (arena_bytes < n->arena_bytes) return fail(TDC_ERR_WORKSPACE, "arena of %zu bytes, %zu are needed", arena_bytes, n->arena_bytes);
    if (reinterpret_cast<uintptr_t>(r.arena) % 16) return fail(TDC_ERR_UNSUPPORTED, "the arena is 16-byte aligned");
    const OnDevice here(n->device);
    for (const auto& op : n->ops) {
        const int rc = op(r);
        if (rc) return rc;               // the step has said why
    }
    return TDC_OK;
}

int tdc_net_run(const tdc_net* n, const float* x, const float* x_absmax, float* y, float* y_absmax, void* arena, size_t arena_bytes, void* stream) {
    return run(n, RunArgs{static_cast<char*>(arena), x, x_absmax, y, y_absmax, (cudaStream_t)stream, false, nullptr, nullptr}, arena_bytes);
}

int tdc_net_run_scaled(const tdc_net* n, const float* x, const float* x_absmax, const float* scale, const float* bias, float* y, float* y_absmax, void* arena, size_t arena_bytes, void* stream) {
    return run(n, RunArgs{static_cast<char*>(arena), x, x_absmax, y, y_absmax, (cudaStream_t)stream, true, scale, bias}, arena_bytes);
}

}  // extern "C"
