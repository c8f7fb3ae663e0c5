"""Convolutions, pooling and the head on packed activations (tdc_net_*), each against the same arithmetic in fp64.

The bar is that of a single layer with fp32-level operands (FP32_TOL): both operands are split into two fp16 parts that carry
22 bits, products of the two lo parts (2^-22) are left out, sums are fp32."""
import os
import subprocess
import sys

import pytest
import torch
import torch.nn.functional as F

from helpers import FP32_TOL, ROOT

pytestmark = pytest.mark.gpu

TILES = [(32, 1, 0), (32, 2, 0), (64, 1, 0), (64, 2, 0), (128, 1, 0), (128, 2, 0), (32, 1, 1), (32, 1, 2), (32, 1, 4), (32, 1, 8), (64, 1, 1), (64, 1, 2), (64, 1, 8)]


@pytest.fixture(scope="module")
def N(built):
    from tdc_b200 import net
    assert torch.cuda.is_available()
    return net


def rel(y, ref):
    return float((y.double() - ref).abs().max() / ref.abs().max())


def draw(seed, B, C, K, H, W, R):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(B, C, H, W, generator=g).cuda()
    w = (torch.randn(K, C, R, R, generator=g) * (2.0 / (K * R * R)) ** 0.5).cuda()
    return x, w, (torch.rand(K, generator=g) + 0.5).cuda(), torch.randn(K, generator=g).cuda()


def conv64(x, w, stride, scale, bias, relu):
    y = F.conv2d(x.double(), w.double(), None, stride, w.shape[2] // 2)
    y = y * scale.double().view(1, -1, 1, 1) + bias.double().view(1, -1, 1, 1)
    return y.relu() if relu else y


# (kind, filter, stride, packing): every form the kernels are instantiated for
KINDS = {"1x1": (0, 1, 1, 0), "3x3": (1, 3, 1, 0), "3x3s2": (2, 3, 2, 1), "7x7s2": (3, 7, 2, 2), "rows": (4, 3, 1, 3), "1x1s2": (5, 1, 2, 1)}


@pytest.mark.parametrize("name", sorted(KINDS))
@pytest.mark.parametrize("B,C,K,H,W", [(2, 40, 72, 13, 11), (1, 200, 130, 7, 9), (3, 3, 5, 16, 18), (150, 17, 33, 7, 7)])
def test_every_kernel_instance(N, name, B, C, K, H, W):
    """Ragged channels, odd images, one tile and several per CTA, more ranks than channel blocks; every instance that fits."""
    from tdc_b200 import TdcError, tc
    kind, R, stride, pack = KINDS[name]
    if name in ("7x7s2", "rows"):
        C = min(C, 5)
    x, w, scale, bias = draw(11 * B + K, B, C, K, H, W, R)
    ref = conv64(x, w, stride, scale, bias, True)
    ran = 0
    for tile in TILES + [None]:
        net = N.Net(B, C, H, W, x.device)
        try:
            net.conv(net.pack(pack), kind, w, scale, bias, True, out=N.NCHW, tile=tile)
        except TdcError as e:
            assert tile is not None, e          # an instance may not fit; the choice of the library always does
            continue
        y = net.finish(ref.shape)(x)
        assert rel(y, ref) <= FP32_TOL, (tile, rel(y, ref))
        ran += 1
    assert ran >= 8 and tc.status() == 0


@pytest.mark.parametrize("tile", [(32, 1, 0), (64, 2, 0), (128, 1, 0), (32, 1, 4), (64, 1, 1)])
@pytest.mark.parametrize("H,W", [(14, 14), (9, 11)])
def test_chain_with_residual_split_and_planes(N, tile, H, W):
    """What a network strings together: 1x1 with planes, 3x3 with residual and split output (odd and even images), a stride-2
    convolution and a stride-2 shortcut on it, max pooling, head."""
    from tdc_b200 import tc
    B, C, K = 3, 24, 40
    x, w1, s1, b1 = draw(5, B, C, K, H, W, 1)
    _, w2, s2, b2 = draw(6, B, K, K, H, W, 3)
    _, w3, s3, b3 = draw(7, B, K, 56, H, W, 3)
    _, w4, s4, b4 = draw(8, B, K, 56, H, W, 1)
    fc, fb = torch.randn(10, 56, device="cuda"), torch.randn(10, device="cuda")
    net = N.Net(B, C, H, W, x.device)
    a = net.conv(net.pack(), N.CONV1x1, w1, s1, b1, True, out=N.PACKED | N.PLANES, tile=tile)
    b = net.conv(a, N.CONV3x3, w2, s2, b2, True, residual=a, out=N.PACKED, split=True, tile=tile)
    d = net.conv(b, N.CONV1x1_S2, w4, s4, b4, False, out=N.PLANES, tile=tile)
    c = net.conv(b, N.CONV3x3_S2, w3, s3, b3, True, residual=d, out=N.PLANES, tile=tile)
    p = net.pool(c, 3, 2, 1, out=N.PLANES)
    net.head(p, fc, fb)
    net.finish((B, 10))
    ra = conv64(x, w1, 1, s1, b1, True)
    rb = (conv64(ra, w2, 1, s2, b2, False) + ra).relu()
    rc = (conv64(rb, w3, 2, s3, b3, False) + conv64(rb, w4, 2, s4, b4, False)).relu()
    ref = F.max_pool2d(rc, 3, 2, 1).mean((2, 3)) @ fc.double().t() + fb.double()
    for _ in range(2):          # the second run finds the first one's data in its arena
        assert rel(net(x), ref) <= FP32_TOL
    assert tc.status() == 0


@pytest.mark.parametrize("name,pool,nt,B,C,K,H,W", [
    ("3x3", 2, 64, 2, 20, 40, 9, 130),        # odd height, a second tile per row that holds one column pair
    ("3x3", 2, 128, 1, 33, 100, 6, 129),      # odd width
    ("3x3", 2, 64, 40, 16, 64, 16, 12),       # several tiles per CTA
    ("1x1", 2, 64, 3, 70, 50, 5, 64),
    ("1x1", 2, 128, 150, 24, 128, 8, 32),
    ("7x7s2", 3, 64, 2, 3, 64, 33, 37),       # odd feature map: the last window's lower row and right column lie outside
    ("7x7s2", 3, 64, 1, 3, 50, 20, 256),      # a full row of 128, as few tiles as CTAs (every one brings the row above along)
    ("7x7s2", 3, 64, 30, 2, 33, 42, 140),     # CTAs that begin and end inside an image
])
@pytest.mark.parametrize("out", [1, 2, 3])
def test_convolution_that_pools(N, name, pool, nt, B, C, K, H, W, out):
    """Max pooling by the convolution's epilogue, read back through a 1x1 convolution or the head."""
    from tdc_b200 import tc
    kind, R, stride, pack = KINDS[name]
    x, w, scale, bias = draw(B + K + W, B, C, K, H, W, R)
    scale[::3] *= -1                          # (a maximum taken before the scale would show)
    net = N.Net(B, C, H, W, x.device)
    t = net.conv(net.pack(pack), kind, w, scale, bias, True, out=out, pool=pool, tile=(nt, 2, 0))
    ref = F.max_pool2d(conv64(x, w, stride, scale, bias, True), pool, 2, pool // 3)
    if out & N.PACKED:
        w2 = torch.randn(24, K, 1, 1, device="cuda") / K ** 0.5
        net.conv(t, N.CONV1x1, w2, out=N.NCHW)
        ref = F.conv2d(ref, w2.double())
    else:
        fc, fb = torch.randn(10, K, device="cuda"), torch.randn(10, device="cuda")
        net.head(t, fc, fb)
        ref = ref.mean((2, 3)) @ fc.double().t() + fb.double()
    net.finish(ref.shape)
    for _ in range(2):
        assert rel(net(x), ref) <= FP32_TOL
    assert tc.status() == 0


@pytest.mark.parametrize("B,C,K,H,W", [(64, 32, 64, 112, 112), (33, 16, 128, 111, 97), (150, 40, 32, 56, 56), (34, 32, 200, 28, 28)])
def test_last_round_of_single_position_tiles(N, B, C, K, H, W):
    """Short sums, many rounds, slow stores: the groups that drain the accumulators run ahead of each other, and in the last
    round those of the second position tile go over to the first.  One position tile per CTA adds the same products in the
    same order, so the results are equal."""
    x, w, scale, bias = draw(B, B, C, K, H, W, 1)
    ys = []
    for mt in (1, 2, 2, 2):
        net = N.Net(B, C, H, W, x.device)
        net.conv(net.pack(), N.CONV1x1, w, scale, bias, True, out=N.NCHW, tile=(min(K, 64), mt, 0))
        ys.append(net.finish((B, K, H, W))(x))
    assert all(torch.equal(ys[0], y) for y in ys[1:])


@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("B,C,H,W", [(2, 20, 9, 10), (1, 64, 14, 14)])
def test_batchnorm_relu_average_into_one_buffer(N, k, B, C, H, W):
    """The pieces of a dense block: channel ranges of one fp32-plane tensor, read back through BatchNorm + ReLU (+ average)."""
    x, w1, s1, b1 = draw(3, B, C, 32, H, W, 1)
    _, w2, s2, b2 = draw(4, B, C, 16, H, W, 3)
    net = N.Net(B, C, H, W, x.device)
    t = net.pack()
    buf = net.planes(B, 48, H, W)
    net.conv(t, N.CONV1x1, w1, s1, b1, out=N.PLANES, into=buf, into_c=0)
    net.conv(t, N.CONV3x3, w2, s2, b2, out=N.PLANES, into=buf, into_c=32)
    scale, shift = torch.randn(48, device="cuda"), torch.randn(48, device="cuda")
    a = net.pool(buf, k, k, out=N.PACKED, scale=scale, shift=shift, bound=torch.stack([scale.abs().max(), shift.abs().max()]))
    w3 = torch.randn(24, 48, 1, 1, device="cuda")
    net.conv(a, N.CONV1x1, w3, out=N.NCHW)
    z = torch.cat([conv64(x, w1, 1, s1, b1, False), conv64(x, w2, 1, s2, b2, False)], 1)
    z = (z * scale.double().view(1, -1, 1, 1) + shift.double().view(1, -1, 1, 1)).relu()
    ref = F.conv2d(F.avg_pool2d(z, 2, 2) if k == 2 else z, w3.double())
    assert rel(net.finish(ref.shape)(x), ref) <= FP32_TOL


@pytest.mark.parametrize("B,C,N_", [(1, 64, 1000), (5, 37, 11), (16, 512, 1000), (40, 50, 33)])
def test_head(N, B, C, N_):
    x, w, _, _ = draw(9, B, C, C, 7, 5, 1)
    fc, fb = torch.randn(N_, C, device="cuda"), torch.randn(N_, device="cuda")
    net = N.Net(B, C, 7, 5, x.device)
    net.head(net.conv(net.pack(), N.CONV1x1, w, out=N.PLANES), fc, fb)
    ref = F.conv2d(x.double(), w.double()).mean((2, 3)) @ fc.double().t() + fb.double()
    assert rel(net.finish(ref.shape)(x), ref) <= FP32_TOL


def test_range_and_integers(N):
    """Inputs of any magnitude give the same relative error, a value the range sample missed is inside the headroom, and sums
    of small integers stay exact without the loss compensation."""
    x, w, scale, bias = draw(12, 4, 64, 64, 28, 28, 3)
    zero = torch.zeros(64, device="cuda")
    one = torch.ones(64, device="cuda")

    def run(x, w, unbiased=True):
        net = N.Net(*x.shape, x.device)
        y = net.conv(net.pack(), N.CONV3x3, w, unbiased=unbiased, out=N.PACKED)
        eye = torch.eye(64, device="cuda").view(64, 64, 1, 1).contiguous()
        net.conv(y, N.CONV1x1, eye, unbiased=unbiased, out=N.NCHW)
        return net.finish((x.shape[0], 64, 28, 28))(x)
    ref = conv64(x, w, 1, one, zero, False)
    for sx, sw in ((1.0, 1.0), (1e-6, 1.0), (1e20, 1e-9), (3e4, 7e3)):
        assert rel(run(x * sx, w * sw), ref * (sx * sw)) <= FP32_TOL
    xo = x.clone()
    xo.view(-1)[12345] = 100.0 * float(x.abs().max())
    assert rel(run(xo, w), conv64(xo, w, 1, one, zero, False)) <= FP32_TOL
    xi = torch.randint(0, 10, x.shape, generator=torch.Generator().manual_seed(1)).float().cuda()
    assert torch.equal(run(xi, torch.ones_like(w), False).double(), conv64(xi, torch.ones_like(w), 1, one, zero, False))


def test_networks_notice_changes(N):
    """A network's net is rebuilt when a weight is written to or replaced, a hook makes the network run layer by layer."""
    import tdc_b200 as T
    m = T.fill_deterministic(T.tkc_resnet18(precision="auto").eval(), seed=0).cuda()
    ref = T.fill_deterministic(T.tkc_resnet18(precision="fp32").eval(), seed=0).cuda()
    x = torch.randn(2, 3, 96, 64, generator=torch.Generator().manual_seed(2)).cuda()

    def same():
        return rel(m(x), ref(x).double()) <= FP32_TOL
    with torch.no_grad():
        assert same() and any(m._nets.nets.values())
        for net in (m, ref):
            net.layer2[0].conv1.core_kernel.mul_(1.5)
        assert same()
        for net in (m, ref):
            net.layer1[1].bn2.weight = torch.nn.Parameter(net.layer1[1].bn2.weight * 0.5)
        assert same()
        seen = []
        h = m.layer3[0].register_forward_hook(lambda *a: seen.append(1))
        assert same() and seen
        h.remove()
        assert same() and len(seen) == 1


@pytest.mark.parametrize("B,C,K,H,W,stride", [(1, 32, 24, 14, 14, 1), (5, 24, 40, 9, 11, 2), (2, 64, 64, 28, 28, 2)])
@pytest.mark.parametrize("precision", ["auto", "fp16x3"])
def test_tucker_module(N, B, C, K, H, W, stride, precision):
    import tdc_b200 as T

    class HP:
        ranks = {"l": [K // 2, C // 2]}
    torch.manual_seed(4)
    m = T.TKConv2dC_B200(C, K, 3, stride=stride, padding=1, bias=True, hp_dict=HP, name="l").cuda()
    m.bias.data.normal_()
    x = torch.randn(B, C, H, W, device="cuda")
    ref = F.conv2d(F.conv2d(F.conv2d(x.double(), m.first_kernel.double()), m.core_kernel.double(), None, stride, 1), m.last_kernel.double(), m.bias.double())
    m.precision = precision
    with torch.no_grad():
        assert rel(m(x), ref) <= FP32_TOL
        m.last_kernel.mul_(2.0)
        assert rel(m(x), 2 * (ref - m.bias.double().view(1, -1, 1, 1)) + m.bias.double().view(1, -1, 1, 1)) <= FP32_TOL


@pytest.mark.parametrize("R,stride", [(1, 1), (3, 1), (3, 2), (7, 2)])
def test_tcconv_packed_form(N, R, stride):
    """TcConv with the packed form forced: the same convolution as its one-launch form, and the recorded magnitude is the true one."""
    import tdc_b200 as T
    x, w, scale, bias = draw(21, 3, 3 if R == 7 else 24, 40, 20, 18, R)
    conv = T.TcConv(w, mode=4, general=stride > 1)
    kw = dict(stride=stride, padding=R // 2) if stride > 1 else {}
    ref = conv64(x, w, stride, scale, bias, True)
    for packed in (True, False):
        conv.packed = packed
        y = conv(x, scale, bias, None, True, **kw)
        assert rel(y, ref) <= FP32_TOL and float(y._tdc_absmax.max()) == float(y.abs().max())


@pytest.mark.parametrize("precision", ["fp32", "tf32x3", "tf32"])
@pytest.mark.parametrize("net", ["tkc_resnet18", "tkc_resnet50", "tkc_vgg16", "tkc_densenet121"])
def test_nchw_nets_equal_the_layers(N, net, precision):
    """The networks on NCHW tensors make the calls of their layer-by-layer forward from native code: the same features, and
    logits that differ by the rounding of the pooled averages and the classifier's sums (fp32, up to 2048 terms)."""
    import tdc_b200 as T
    m = T.fill_deterministic(getattr(T, net)(precision=precision).eval(), seed=0, gain=0.7 if "dense" in net else 1.0).cuda()
    x = torch.randn(2, 3, 96, 70, generator=torch.Generator().manual_seed(3)).cuda()
    with torch.no_grad():
        y = m(x)
        assert any(m._nets.nets.values())
        h = m.features[0].register_forward_hook(lambda *a: None) if hasattr(m, "features") else m.bn1.register_forward_hook(lambda *a: None)
        ref = m(x)                               # a hook makes the network run layer by layer
        h.remove()
    assert rel(y, ref.double()) <= FP32_TOL


OVERFLOW = """
import sys
for p in sys.argv[1:3]:
    sys.path.insert(0, p)
import torch
import tdc_b200 as T
from tdc_b200 import net as N, tc
kind, R, pack, pool, tile, C, K, H, W = eval(sys.argv[3])
g = torch.Generator().manual_seed(1)
x = torch.randn(2, C, H, W, generator=g).cuda()
w = torch.randn(K, C, R, R, generator=g).cuda()


def run(x):
    net = N.Net(*x.shape, x.device)
    t = net.conv(net.pack(pack), kind, w, relu=True, out=N.PLANES if pool else N.NCHW, pool=pool, tile=tile)
    if pool:
        net.head(t, torch.eye(K, device="cuda"), None)
        return net.finish((2, K))(x)
    return net.finish((2, K, H, W))(x)


assert bool(run(x).isfinite().all()) and tc.status() == 0
x[1, 0, H // 2, W // 2] = 1e5 * float(x.abs().max())
y = run(x)
assert bool(y[0].isfinite().all()) and not bool(y[1].isfinite().all()), y
assert tc.status() == 2
x = torch.randn(2, 16, 56, 56, generator=g).cuda()
x[1, 0, 5, 3] = 1e5 * float(x.abs().max())      # (element 50459: that kernel's sample takes every 49th)
conv = T.TcConv(torch.randn(K, 16, 3, 3, generator=g).cuda(), mode=4)
conv.packed = False
assert not bool(conv(x, relu=True)[1].isfinite().all())
"""


@pytest.mark.parametrize("case", [(1, 3, 0, 0, (64, 2, 0), 32, 64, 72, 72), (1, 3, 0, 0, (32, 1, 4), 512, 32, 24, 24), (0, 1, 0, 0, (32, 1, 1), 64, 32, 50, 50),
                                  (1, 3, 0, 2, (64, 2, 0), 32, 64, 72, 72), (3, 7, 2, 3, (64, 2, 0), 3, 64, 240, 240), (4, 3, 3, 0, (64, 1, 0), 3, 64, 240, 240)])
def test_overflow_is_reported_behind_relu_and_pooling(N, case):
    """A value beyond 256 times the sampled maximum (inputs of more than 2^18 values are sampled): the outputs that read it are not finite, ReLU and maxima included, and the status
    word says 2 (in a process of its own, because the word keeps its first report)."""
    r = subprocess.run([sys.executable, "-c", OVERFLOW, os.path.join(ROOT, "ppopp23-tdc_b200"), ROOT, repr(case)], capture_output=True, text=True,
                       env=dict(os.environ, TDC_TC_TUNING="0"), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("B,C,H,W", [(16, 3, 224, 224), (2, 16, 100, 125)])
def test_range_sample_is_spread(N, B, C, H, W):
    """Values at a fixed distance would all lie in the first columns of a batch of 16 images (and in the first image of a small batch),
    which are a thousandth of the rest here: the sample has to see the others."""
    from tdc_b200 import tc
    x = torch.randn(B, C, H, W, generator=torch.Generator().manual_seed(1))
    x[:, :, :, 0] *= 1e-3
    if B == 2:
        x[0] *= 1e-3
    x = x.cuda()
    w = (torch.randn(8, C, 3, 3, generator=torch.Generator().manual_seed(2)) * 0.1).cuda()
    net = N.Net(B, C, H, W, x.device)
    net.conv(net.pack(), N.CONV3x3, w, relu=True, out=N.NCHW)
    y = net.finish((B, 8, H, W))(x)
    assert rel(y, F.conv2d(x.double(), w.double(), None, 1, 1).relu()) <= FP32_TOL and tc.status() == 0


@pytest.mark.parametrize("what", ["network", "module", "layer"])
def test_built_on_one_stream_run_on_another(N, what):
    """What a net was built from is ready before any stream's run reads it, and stays while one reads it: the build waits behind a
    long kernel, the run is another stream's; then the filters are replaced and their memory is asked for and written while
    that stream has not come to its run yet."""
    import tdc_b200 as T

    class HP:
        ranks = {"l": [32, 32]}
    torch.manual_seed(5)
    if what == "network":
        m, x = T.fill_deterministic(T.tkc_resnet18(precision="auto").eval(), seed=0).cuda(), torch.randn(2, 3, 96, 64, device="cuda")
        weight = m.layer2[0].conv1.core_kernel
    elif what == "module":
        m, x = T.TKConv2dC_B200(64, 64, 3, padding=1, hp_dict=HP, name="l").cuda(), torch.randn(2, 64, 14, 14, device="cuda")
        m.precision, weight = "fp16x3", m.core_kernel
    else:
        m, x = T.TcConv(torch.randn(64, 64, 3, 3, device="cuda"), mode=4), torch.randn(2, 64, 14, 14, device="cuda")
        m.packed, weight = True, None
    ref = None
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.no_grad():
        for repeat in range(2):
            torch.cuda.synchronize()
            with torch.cuda.stream(a):
                torch.cuda._sleep(100_000_000)
                m(x)
            with torch.cuda.stream(b):
                y = m(x)
                torch.cuda._sleep(100_000_000)
                late = m(x)
            if weight is not None:
                with torch.cuda.stream(a):
                    weight.mul_(1.0)             # another version: the next call prepares the filters anew
                    m(x)
                    junk = [torch.full((n,), float("nan"), device="cuda") for n in (1 << 12, 1 << 14, 1 << 16, 1 << 18, 1 << 20) for _ in range(8)]
                    del junk
            torch.cuda.synchronize()
            ref = m(x) if ref is None else ref
            torch.cuda.synchronize()
            assert bool(ref.isfinite().all()) and torch.equal(y, ref) and torch.equal(late, ref)


@pytest.mark.parametrize("R,stride", [(1, 1), (3, 2)])
def test_scale_and_bias_come_with_the_call(N, R, stride):
    """One net per shape, whatever vectors a call brings: new ones on every call, one of the two, none, and the same memory rewritten."""
    import tdc_b200 as T
    x, w, scale, bias = draw(22, 2, 24, 40, 15, 13, R)
    conv = T.TcConv(w, mode=4, general=stride > 1)
    conv.packed = True
    kw = dict(stride=stride, padding=R // 2) if stride > 1 else {}
    one, zero = torch.ones_like(scale), torch.zeros_like(bias)
    for k in range(4):
        s, b = scale * (k + 1), bias - k
        for sc, bi in ((s, b), (s, None), (None, b), (None, None)):
            ref = conv64(x, w, stride, one if sc is None else sc, zero if bi is None else bi, True)
            assert rel(conv(x, sc, bi, None, True, **kw), ref) <= FP32_TOL
    s = scale.clone()
    for _ in range(2):
        assert rel(conv(x, s, bias, None, True, **kw), conv64(x, w, stride, s, bias, True)) <= FP32_TOL
        s.mul_(-2.0)
    assert len(conv._nets) == 1


@pytest.mark.parametrize("C,H,mode", [(64, 14, 4), (256, 7, 4), (64, 56, 4), (64, 14, 3)])
def test_layer_is_that_of_its_weight_when_it_was_made(N, monkeypatch, C, H, mode):
    """Forms prepared when a shape first needs them (packed, other block sizes) are those of the weight at construction, and the
    layer's switches count on every call."""
    import tdc_b200 as T
    from tdc_b200 import tc
    monkeypatch.setattr(tc, "_TUNING", False)
    x, w, _, _ = draw(23, 2, C, C, H, H, 3)
    one, zero = torch.ones(C, device="cuda"), torch.zeros(C, device="cuda")
    conv, ref = T.TcConv(w, mode=mode), conv64(x, w, 1, one, zero, False)
    fresh = {u: T.TcConv(w.clone(), mode=mode, unbiased=u) for u in (False, True)}
    w.mul_(3.0)
    for B in (2, 1, 2):
        assert rel(conv(x[:B]), ref[:B]) <= FP32_TOL
    for unbiased in (True, False):
        conv.unbiased = unbiased
        assert torch.equal(conv(x), fresh[unbiased](x))
    conv.exact_range = mode == 4
    assert rel(conv(x), ref) <= FP32_TOL


def test_modules_pass_their_range_on(N):
    """The exact range goes from layer to module to module: a value far beyond what a sample would see stays in the headroom of none.
    A tensor that was written to since is sampled."""
    import tdc_b200 as T
    from tdc_b200 import tc

    class HP:
        ranks = {"l": [16, 16]}
    torch.manual_seed(6)
    C, H = 32, 80
    first = T.TcConv(torch.randn(C, C, 1, 1, device="cuda"), mode=4, exact_range=True)
    for precision in ("auto", "fp16x3"):
        m = T.TKConv2dC_B200(C, C, 3, padding=1, bias=False, hp_dict=HP, name="l").cuda()
        m.precision = precision
        x = torch.randn(2, C, H, H, device="cuda")
        x[1, 3, 7, 9] = 1e5 * float(x.abs().max())

        def tucker(x):
            return F.conv2d(F.conv2d(F.conv2d(x.double(), m.first_kernel.double()), m.core_kernel.double(), None, 1, 1), m.last_kernel.double())
        with torch.no_grad():
            y = first(x)
            z = m(m(y))
            assert rel(z, tucker(tucker(y))) <= FP32_TOL and tc.status() == 0
            assert precision == "auto" or float(z._tdc_absmax.max()) == float(z.abs().max())      # ("auto" ends in fp32 here)
            y = m(torch.randn(2, C, H, H, device="cuda"))
            y.mul_(1e6)                                 # what it carries is no bound any more
            assert rel(m(y), tucker(y)) <= FP32_TOL and tc.status() == 0


@pytest.mark.parametrize("B,C,affine", [(1, 64, False), (5, 37, True), (40, 50, False)])
def test_averages_without_a_classifier(N, B, C, affine):
    x, w, s, b = draw(9, B, C, C, 7, 5, 1)
    net = N.Net(B, C, 7, 5, x.device)
    net.head(net.conv(net.pack(), N.CONV1x1, w, out=N.PLANES), None, None, *((s, b) if affine else (None, None)))
    ref = F.conv2d(x.double(), w.double())
    if affine:
        ref = (ref * s.double().view(1, -1, 1, 1) + b.double().view(1, -1, 1, 1)).relu()
    assert rel(net.finish((B, C))(x), ref.mean((2, 3))) <= FP32_TOL


@pytest.mark.parametrize("net", ["tkc_resnet18", "tkc_densenet121"])
@pytest.mark.parametrize("precision", ["auto", "fp32"])
def test_classifier_is_trained_on_a_frozen_network(N, net, precision):
    """The gradient of the classifier is that of torch's Linear on the network's averages; the logits are those of the net's own."""
    import tdc_b200 as T
    m = T.fill_deterministic(getattr(T, net)(precision=precision).eval(), seed=0, gain=0.7 if "dense" in net else 1.0).cuda()
    fc = m.fc if hasattr(m, "fc") else m.classifier
    x = torch.randn(2, 3, 96, 64, generator=torch.Generator().manual_seed(2)).cuda()
    y = m(x)
    g = torch.randn_like(y)
    y.backward(g)
    with torch.no_grad():
        assert rel(m(x), y.double().detach()) <= FP32_TOL and any(n and not n.features for n in m._nets.nets.values())
        seen = []
        h = fc.register_forward_hook(lambda mod, a, out: seen.append(a[0]))
        m(x)
        h.remove()
    assert rel(fc.weight.grad, g.double().t() @ seen[0].double()) <= FP32_TOL and torch.allclose(fc.bias.grad, g.sum(0))


@pytest.mark.parametrize("R,general,kw,H,W", [(3, False, {"stride": 2}, 12, 12), (3, False, {}, 4, 300), (1, False, {}, 4, 300), (3, True, {"stride": 2, "padding": 1}, 4, 600)])
def test_packed_form_takes_no_call_the_layer_refuses(N, monkeypatch, R, general, kw, H, W):
    """A stride without a general plan, an image wider than a plan's 256 positions."""
    import tdc_b200 as T
    from tdc_b200 import tc
    monkeypatch.setattr(tc, "_TUNING", False)
    x, w, _, _ = draw(24, 1, 16, 24, H, W, R)
    codes = []
    for packed in (False, True, None):
        conv = T.TcConv(w, mode=4, general=general)
        conv.packed = packed
        try:
            conv(x, **kw)
            codes.append(0)
        except T.TdcError as e:
            codes.append(e.code)
    assert codes[0] == codes[1] == codes[2] and codes[0] in (0, 2, 3, 5)


@pytest.mark.parametrize("pack", [0, 1, 2, 3])
@pytest.mark.parametrize("B,C,H,W", [(1, 3, 17, 19), (2, 20, 33, 40), (1, 64, 64, 64), (5, 1, 200, 250), (1, 5, 3, 3)])
def test_small_inputs_have_their_true_range(N, pack, B, C, H, W):
    """Up to 2^18 values the packing pass finds the true maximum: any value anywhere keeps its bits, from the first to the last
    element, aligned or not; beside it the ordinary values keep those of fp32 sums."""
    from tdc_b200 import tc
    kind, R, stride, _ = KINDS[{0: "3x3", 1: "3x3s2", 2: "7x7s2", 3: "rows"}[pack]]
    if pack >= 2:
        C = min(C, 5)
    x0, w, scale, bias = draw(31, B, C, 24, H, W, R)
    room = torch.empty(x0.numel() + 1, device="cuda")
    for at, off in ((0, 0), (x0.numel() - 1, 1), (x0.numel() // 2 + 1, 0)):
        x = room[off:off + x0.numel()].view_as(x0).copy_(x0)
        x.view(-1)[at] = 1e7
        net = N.Net(B, C, H, W, x.device)
        net.conv(net.pack(pack), kind, w, scale, bias, True, out=N.NCHW)
        ref = conv64(x, w, stride, scale, bias, True)
        y = net.finish(ref.shape)(x)
        assert rel(y, ref) <= FP32_TOL and tc.status() == 0
        away = (F.conv2d((x == 1e7).double(), torch.ones(24, C, R, R, device="cuda").double(), None, stride, R // 2) == 0).double()
        assert float(((y - ref) * away).abs().max()) <= FP32_TOL * max(1.0, float((ref * away).abs().max()))


@pytest.mark.parametrize("B,C,R1,H,stride", [(1, 64, 32, 14, 1), (1, 64, 32, 14, 2), (2, 512, 8, 32, 1), (2, 512, 8, 32, 2)])
def test_auto_modules_take_any_value_where_they_began_in_fp32(N, B, C, R1, H, stride):
    """Layers below the size from which "auto" used tensor cores have no range: small inputs are packed with their true one, larger ones
    after a pass that finds it."""
    import tdc_b200 as T
    from tdc_b200 import dispatch, tc

    class HP:
        ranks = {"l": [32, R1]}
    torch.manual_seed(7)
    m = T.TKConv2dC_B200(C, 64, 3, stride=stride, padding=1, bias=False, hp_dict=HP, name="l").cuda()
    m.precision = "auto"
    x = torch.randn(B, C, H, H, device="cuda")
    assert not dispatch._on_tensor_cores(B, C, R1, H, H, 1, 1, 1, 0)
    x[-1, 1, 3, 5] = 1e6
    ref = F.conv2d(F.conv2d(F.conv2d(x.double(), m.first_kernel.double()), m.core_kernel.double(), None, stride, 1), m.last_kernel.double())
    with torch.no_grad():
        assert rel(m(x), ref) <= FP32_TOL and tc.status() == 0
