"""Whole networks as nets: on packed activations under "auto" and "fp16x3", as the layer-by-layer kernels on NCHW tensors
under the other precisions.

A network's forward is looked up by input shape; the first call of a shape builds the net (net.Net) from the modules, later
calls run it with one library call.  The modules stay what they are — parameters, state dict, submodules — and what a net
was built from is compared with them on every call, AFTER the launches are issued, so that the comparison costs no latency:
where something changed (a weight written to or replaced, a submodule exchanged, a hook registered) the nets are dropped and
the forward runs again.  A network that a net cannot express (an exotic stride, a hook that wants to see a layer) runs
layer by layer.  So does one with a module of another kind in a place that the layer-by-layer forward CALLS (stages, blocks, the
average pool, the classifier): a net stands for the forwards of the exact classes named in the builders, no subclass's."""
import functools
import math
import threading

import torch
import torch.nn as nn
from torch.autograd import forward_ad
from torch.nn.modules import module as _module

from . import net as N
from ._lib import ERR_SHAPE, ERR_SMEM, ERR_UNSUPPORTED, NetConv, TdcError, check, lib
from .ops import ABSMAX_FLOATS, _stream, range_of

import ctypes as C

PRECISIONS = ("auto", "fp16x3")                  # on packed activations
NCHW_PRECISIONS = ("fp32", "tf32x3", "tf32")     # the layer-by-layer kernels, launched from native code


class NotExpressible(Exception):
    """This network or layer is no chain of the launches a net has."""


def _exact(module, *kinds):
    """`module`, if its forward is the one of these classes that a net stands for."""
    if type(module) not in kinds:
        raise NotExpressible
    return module


def _average_to_one(pool):
    if _exact(pool, nn.AdaptiveAvgPool2d).output_size not in (1, (1, 1), [1, 1]):
        raise NotExpressible


# ---- BatchNorm folding -----------------------------------------------------------------------------------------------
def fold_bn(bn):
    """(scale, shift, {max |scale|, max |shift|}) of an inference BatchNorm on the GPU, kept on the module until one of its
    tensors changes."""
    key = (bn.eps,) + N._key(bn.running_var, bn.running_mean, bn.weight, bn.bias)
    kept = bn.__dict__.setdefault("_tdc_fold", N.Cache())
    hit = kept.get("fold")
    if hit is None or hit[0] != key:
        tensors = (bn.running_var, bn.running_mean, bn.weight, bn.bias)
        n, dev = bn.running_var.numel(), bn.running_var.device
        n4 = (n + 3) // 4 * 4                                 # scale and shift 16-byte aligned
        buf = torch.empty(2 * n4 + 2, device=dev, dtype=torch.float32)
        scale, shift, bound = buf[:n], buf[n4:n4 + n], buf[2 * n4:]
        with N.building(dev):
            N.building.made()
            if all(t is None or (t.dtype == torch.float32 and t.is_contiguous() and t.device == dev and t.numel() == n) for t in tensors):
                var, mean, g, b = (None if t is None else t.data_ptr() for t in tensors)
                check(lib.tdc_net_fold_bn(var, mean, g, b, bn.eps, n, scale.data_ptr(), shift.data_ptr(), bound.data_ptr(), _stream()))
            else:                                             # another type or layout: the same arithmetic
                with torch.no_grad():
                    var, mean = bn.running_var.double(), bn.running_mean.double()
                    s = (1.0 if bn.weight is None else bn.weight.double()) / torch.sqrt(var + bn.eps)
                    scale.copy_(s), shift.copy_((0.0 if bn.bias is None else bn.bias.double()) - mean * s)
                    bound.copy_(torch.stack([scale.abs().max(), shift.abs().max()]))
        hit = kept["fold"] = (key, scale, shift, bound)
    return hit[1:]


# ---- one convolution module ------------------------------------------------------------------------------------------
class At:
    """A tensor of the net under construction: number, channels and image."""
    __slots__ = ("id", "C", "H", "W", "split")

    def __init__(self, id, Cc, H, W, split=False):
        self.id, self.C, self.H, self.W, self.split = id, Cc, H, W, split


def _estimate(*layer):
    return _estimate_on(torch.cuda.current_device(), *layer)


def _pooled_estimates(*layer):
    return _pooled_estimates_on(torch.cuda.current_device(), *layer)


# (remembered: a module weighs several forms that share steps, a network repeats its blocks)
@functools.lru_cache(maxsize=8192)
def _estimate_on(device, B, Cc, H, W, split, kind, K, residual, out, pool=0):
    if pool:
        return min(_pooled_estimates_on(device, B, Cc, H, W, split, kind, K, out, pool))
    d = NetConv()
    d.kind, d.K, d.residual, d.out, d.into = kind, K, 0 if residual else -1, out, -1
    check(lib.tdc_net_estimate(B, Cc, H, W, int(split), C.byref(d)))
    return d.clocks


@functools.lru_cache(maxsize=8192)
def _pooled_estimates_on(device, B, Cc, H, W, split, kind, K, out, pool):
    """Clocks of a convolution whose epilogue pools (infinite where no kernel does), and of the two steps one by one: pooling
    reads fp32 planes and leaves `out`, from HBM where it moves more than L2 holds (bytes per clock of the whole chip)."""
    d = NetConv()
    d.kind, d.K, d.residual, d.out, d.into, d.relu, d.pool = kind, K, -1, out, -1, 1, pool
    one = d.clocks if lib.tdc_net_estimate(B, Cc, H, W, int(split), C.byref(d)) == 0 else math.inf
    size = 4.0 * B * K * H * W * (1 + 0.25 * bin(out).count("1"))
    return one, _estimate_on(device, B, Cc, H, W, split, kind, K, False, N.PLANES) + 4000.0 + size / (2600.0 if size > 80e6 else 6500.0)


def _pool_of(m):
    """`pool` of a convolution that does this max pooling itself, or 0."""
    k, s, p, d = ((v, v) if isinstance(v, int) else tuple(v) for v in (m.kernel_size, m.stride, m.padding, m.dilation))
    if m.ceil_mode or d != (1, 1):
        return 0
    return 2 if (k, s, p) == ((2, 2), (2, 2), (0, 0)) else 3 if (k, s, p) == ((3, 3), (2, 2), (1, 1)) else 0


def _square(conv, size):
    """The stride of a "same" convolution of this filter size, or NotExpressible."""
    if tuple(conv.kernel_size) != (size, size) or tuple(conv.padding) != (size // 2, size // 2) or conv.stride[0] != conv.stride[1] \
            or conv.stride[0] not in (1, 2) or tuple(conv.dilation) != (1, 1) or conv.groups != 1:
        raise NotExpressible
    return conv.stride[0]


def _with_bias(conv, scale, shift):
    """(conv + bias) * scale + shift, kept on the module: a captured graph reads it after the net it was captured from has made room
    for another shape's, as it reads the filters and folds kept there."""
    if conv.bias is None:
        return shift
    if scale is None and shift is None:
        return conv.bias.detach()
    key = N._key(conv.bias, scale, shift)
    kept = conv.__dict__.setdefault("_tdc_shift", N.Cache())
    hit = kept.get("shift")
    if hit is None or hit[0] != key:
        N.building.made()
        b = conv.bias.detach() if scale is None else conv.bias.detach() * scale
        hit = kept["shift"] = (key, b if shift is None else shift + b, conv.bias.detach(), scale, shift)
    return hit[1]


def conv(net, module, x, scale, shift, relu, precision, residual=-1, out=N.PACKED, split=False, into=-1, into_c=0, pool=None):
    """`module` (dense, Tucker or SVD) with its epilogue on tensor `x`; returns what it made.  `pool`: a max pooling that follows
    the ReLU; `out` is then the pooled tensor's."""
    from .svdconv import _SVDConvBase
    from .tkconv import TKConv2dC_B200
    if precision in NCHW_PRECISIONS:
        return nchw_conv(net, module, x, scale, shift, relu, precision, residual)
    shift = _with_bias(module, scale, shift)
    end = dict(scale=scale, bias=shift, relu=relu, residual=residual, out=out, split=split, into=into, into_c=into_c)
    pooling = _pool_of(pool) if pool is not None else 0

    def step(src, kind, weight, name, last, K):
        if tuple(weight.shape[:2]) != (K, src.C) or weight.shape[2] != weight.shape[3]:
            raise NotExpressible
        stride = 2 if kind in (N.CONV3x3_S2, N.CONV1x1_S2) else 1
        opts = end if last else {}
        if last and pool is not None:
            one, two = _pooled_estimates(B, src.C, src.H, src.W, src.split, kind, K, out, pooling) if pooling and relu and residual < 0 else (1, 0)
            if one >= two:
                t = net.conv(src.id, kind, weight, owner=module, name=name, **dict(end, out=N.PLANES))
                return pool_max(net, pool, At(t, K, -(-src.H // stride), -(-src.W // stride)), out)()
            t = net.conv(src.id, kind, weight, owner=module, name=name, pool=pooling, **end)
            return At(t, K, _pooled(pool, src.H), _pooled(pool, src.W))
        t = net.conv(src.id, kind, weight, owner=module, name=name, **opts)
        return At(t, K, -(-src.H // stride), -(-src.W // stride), (last and split) or (src.split and stride == 1))

    B = net.shape[0]
    if isinstance(module, _SVDConvBase):
        if tuple(module.dilation) != (1, 1) or tuple(module.padding) != (0, 0) or x.split:
            raise NotExpressible
        left, right = module._kernels()
        z = step(x, N.CONV1x1, left, "left", False, module.rank)
        return step(z, N.CONV1x1, right, "right", True, module.out_channels)
    if isinstance(module, TKConv2dC_B200):
        stride = _square(module, 3)
        core = N.CONV3x3_S2 if stride == 2 else N.CONV3x3
        K, R1, R2 = module.out_channels, module.in_rank, module.out_rank
        Ho, Wo = -(-x.H // stride), -(-x.W // stride)
        form = "chain"
        pooling = pooling if relu and residual < 0 and stride == 1 else 0
        if precision == "auto":
            # the three steps, the last two multiplied into one filter, or all three: the same linear map in fewer, larger
            # launches; whichever the estimates say is the fastest
            first = _estimate(B, x.C, x.H, x.W, x.split, N.CONV1x1, R1, False, N.PACKED)
            cost = {"chain": first + _estimate(B, R1, x.H, x.W, x.split, core, R2, False, N.PACKED)
                    + _estimate(B, R2, Ho, Wo, False, N.CONV1x1, K, residual >= 0, out, pooling),
                    "fold": first + _estimate(B, R1, x.H, x.W, x.split, core, K, residual >= 0, out, pooling),
                    "dense": _estimate(B, x.C, x.H, x.W, x.split, core, K, residual >= 0, out, pooling)}
            form = min(cost, key=cost.get)
        if form == "dense":
            return step(x, core, module._dense_weight(), "dense", True, K)
        z = step(x, N.CONV1x1, module.first_kernel, "first", False, R1)
        if form == "fold":
            return step(z, core, module._core_last_weight(), "core_last", True, K)
        z = step(z, core, module.core_kernel, "core", False, R2)
        return step(z, N.CONV1x1, module.last_kernel, "last", True, K)
    K = module.out_channels
    if tuple(module.kernel_size) == (1, 1):
        stride = _square(module, 1)
        return step(x, N.CONV1x1_S2 if stride == 2 else N.CONV1x1, module.weight, "weight", True, K)
    stride = _square(module, 3)
    return step(x, N.CONV3x3_S2 if stride == 2 else N.CONV3x3, module.weight, "weight", True, K)


def nchw_step(net, owner, name, x, w, scale, shift, relu, precision, residual, stride, pad, to_y=False):
    """One convolution on NCHW tensors: the kernel `dispatch.one_conv` takes for a named precision."""
    from . import dispatch, tc
    K, Cc, R, S = w.shape
    B = net.shape[0]
    if R != S or x.C != Cc or x.H + 2 * pad < R or x.W + 2 * pad < R:
        raise NotExpressible
    Ho, Wo = (x.H + 2 * pad - R) // stride + 1, (x.W + 2 * pad - R) // stride + 1
    one_pass = tc.supported(R, S, stride, pad, x.W)
    if precision != "fp32" and (one_pass or tc.general_supported(R, S, stride, pad, Wo)) and not (precision == "tf32x3" and dispatch._f32_first(B, Cc, K, Ho, Wo, R, S, stride)):
        general = not one_pass or dispatch._thin_and_wide(Cc, x.W, R, stride)
        conv = tc.cached(owner, name, w, dispatch.MODES[precision], general=general)
        plan, flt, flags = conv.step(B, x.H, x.W, stride, pad)
    else:
        plan, flt, flags = None, dispatch.channel_last(owner, name, w), 0
    t = net.nchw_conv(x.id, K, R, stride, pad, flt, scale, shift, residual, relu, plan, flags, to_y=to_y)
    return At(t, K, Ho, Wo)


def nchw_conv(net, module, x, scale, shift, relu, precision, residual=-1):
    """`conv` on NCHW tensors; `shift` has the module's bias in it already when `conv` calls this."""
    from .svdconv import _SVDConvBase
    from .tkconv import TKConv2dC_B200
    if module.stride[0] != module.stride[1] or module.padding[0] != module.padding[1] or tuple(module.dilation) != (1, 1) or module.groups != 1:
        raise NotExpressible
    shift = _with_bias(module, scale, shift)
    stride, pad = module.stride[0], module.padding[0]

    def step(src, name, w, last, st, p):
        return nchw_step(net, module, name, src, w, scale if last else None, shift if last else None, relu and last, precision, residual if last else -1, st, p)
    if isinstance(module, _SVDConvBase):
        if pad:
            raise NotExpressible
        left, right = module._kernels()
        return step(step(x, "left", left, False, 1, 0), "right", right, True, 1, 0)
    if isinstance(module, TKConv2dC_B200):
        z = step(x, "first", module.first_kernel, False, 1, 0)
        return step(step(z, "core", module.core_kernel, False, stride, pad), "last", module.last_kernel, True, 1, 0)
    return step(x, "weight", module.weight, True, stride, pad)


def stem7(net, module, scale, shift, pool, out, precision):
    """The 7x7 stride-2 convolution on the NCHW input, with ReLU, and the max pooling behind it; a callable that takes pool_max's
    options."""
    if precision in NCHW_PRECISIONS:
        return pool_max(net, pool, nchw_conv(net, module, At(-1, *net.shape[1:]), scale, shift, True, precision), out)
    if tuple(module.kernel_size) != (7, 7) or tuple(module.stride) != (2, 2) or tuple(module.padding) != (3, 3) or tuple(module.dilation) != (1, 1) or module.groups != 1:
        raise NotExpressible
    B, Cc, H, W = net.shape
    if Cc != module.weight.shape[1]:
        raise NotExpressible
    t, K, H, W = net.pack(N.PACK_S2D), module.weight.shape[0], -(-H // 2), -(-W // 2)
    opts = dict(scale=scale, bias=_with_bias(module, scale, shift), relu=True, owner=module, name="weight")
    pooling = _pool_of(pool)
    if pooling:
        one, two = _pooled_estimates(B, 4 * Cc, H, W, False, N.CONV7x7_S2, K, out, pooling)
        if one < two:
            return lambda **kw: At(net.conv(t, N.CONV7x7_S2, module.weight, out=out, pool=pooling, **opts, **kw), K, _pooled(pool, H), _pooled(pool, W))
    return pool_max(net, pool, At(net.conv(t, N.CONV7x7_S2, module.weight, out=N.PLANES, **opts), K, H, W), out)


def pool_max(net, m, x, out):
    k, s, p = ((v[0] if isinstance(v, (tuple, list)) else v) for v in (m.kernel_size, m.stride, m.padding))
    if m.ceil_mode or (m.dilation != 1 and m.dilation != (1, 1)) or any(isinstance(v, (tuple, list)) and v[0] != v[1] for v in (m.kernel_size, m.stride, m.padding)):
        raise NotExpressible
    H, W = (x.H + 2 * p - k) // s + 1, (x.W + 2 * p - k) // s + 1
    if H <= 0 or W <= 0:
        raise NotExpressible
    if net.nchw:
        return lambda: At(net.nchw_pool(x.id, k, s, p, 0), x.C, H, W)
    return lambda **kw: At(net.pool(x.id, k, s, p, out=out, **kw), x.C, H, W)


# ---- the classifier ----------------------------------------------------------------------------------------------------
def native_classifier(head, x):
    """What identifies a classifier that a net's last launch stands for, or None where `head` has to be called on the averages:
    another module than a Linear on fp32 memory, hooks, and whatever torch does around a call — gradients, autocast, forward-mode
    derivatives, function transforms, dispatch modes."""
    if type(head) is not nn.Linear or "forward" in head.__dict__ or head._forward_hooks or head._forward_pre_hooks or head._backward_hooks or head._backward_pre_hooks:
        return None
    w, b = head._parameters.get("weight"), head._parameters.get("bias")
    if w is None or (torch.is_grad_enabled() and (w.requires_grad or (b is not None and b.requires_grad))) or torch.is_autocast_enabled(x.device.type) \
            or forward_ad._current_level >= 0 or torch._C._functorch.peek_interpreter_stack() is not None or torch._C._len_torch_dispatch_stack():
        return None
    if any(t is not None and (t.dtype != torch.float32 or t.device != x.device or not t.is_contiguous()) for t in (w, b)):
        return None
    return (w.data_ptr(), None if b is None else b.data_ptr(), w.shape)


def classify(net, x, head, scale=None, shift=None):
    """The end of a network: averages and classifier, or (net.features) the averages that `head` is called on."""
    if net.features:
        net.head(x.id, None, None, scale, shift)
        return net.finish((net.shape[0], x.C))
    net.head(x.id, head.weight, head.bias, scale, shift)
    return net.finish((net.shape[0], head.weight.shape[0]))


# ---- the networks ----------------------------------------------------------------------------------------------------
def build_resnet(model, net, precision):
    from .resnet import TKBasicBlock, TKBottleneck
    _average_to_one(model.avgpool)
    s, b, _ = fold_bn(model.bn1)
    blocks = [_exact(m, TKBasicBlock, TKBottleneck) for layer in (model.layer1, model.layer2, model.layer3, model.layer4) for m in _exact(layer, nn.Sequential)]
    wide = [type(m) is TKBottleneck for m in blocks]

    def strided(i):
        return i < len(blocks) and (blocks[i].conv2 if wide[i] else blocks[i].conv1).stride[0] == 2

    def outputs(i):
        """What the block before block i has to leave: operands, and fp32 planes where block i adds its input to its output."""
        if i == len(blocks):
            return N.PLANES
        return N.PACKED | (0 if blocks[i].downsample is not None else N.PLANES)
    if strided(0):
        raise NotExpressible
    x = stem7(net, model.conv1, s, b, model.maxpool, outputs(0), precision)()
    for i, m in enumerate(blocks):
        s1, b1, _ = fold_bn(m.bn1)
        s2, b2, _ = fold_bn(m.bn2)
        out = conv(net, m.conv1, x, s1, b1, True, precision)
        last = m.conv2
        if wide[i]:
            out = conv(net, m.conv2, out, s2, b2, True, precision)
            s2, b2, _ = fold_bn(m.bn3)
            last = m.conv3
        identity = x
        if m.downsample is not None:
            sd, bd, _ = fold_bn(m.downsample[1])
            identity = conv(net, m.downsample[0], x, sd, bd, False, precision, out=N.PLANES)
        o = outputs(i + 1)
        if strided(i + 1) and o & N.PLANES:
            raise NotExpressible
        x = conv(net, last, out, s2, b2, True, precision, residual=identity.id, out=o, split=strided(i + 1))
    return classify(net, x, model.fc)


def build_vgg(model, net, precision):
    from .resnet import Conv2dB200
    from .vgg import TKVGG
    if type(model).forward_features is not TKVGG.forward_features:
        raise NotExpressible
    mods = list(model.features)
    x, i = None, 0
    B, Cc, H, W = net.shape

    def planes_next(j):
        return N.PLANES if j >= len(mods) or isinstance(mods[j], nn.MaxPool2d) else N.PACKED
    while i < len(mods):
        m = mods[i]
        if isinstance(m, nn.MaxPool2d):
            if x is None:
                raise NotExpressible
            i += 1
            x = pool_max(net, m, x, planes_next(i))()
            continue
        scale = shift = None
        j = i + 1
        if j < len(mods) and isinstance(mods[j], nn.BatchNorm2d):
            scale, shift, _ = fold_bn(mods[j])
            j += 1
        relu = j < len(mods) and isinstance(mods[j], nn.ReLU)
        i = j + (1 if relu else 0)
        out = planes_next(i)
        if x is None and net.nchw:
            x = At(-1, Cc, H, W)
        elif x is None:
            if type(m) is Conv2dB200 and 3 * Cc <= 16 and _square(m, 3) == 1:
                if m.weight.shape[1] != Cc:
                    raise NotExpressible
                t = net.conv(net.pack(N.PACK_ROWS), N.CONV3x3_ROWS, m.weight, scale=scale, bias=_with_bias(m, scale, shift), relu=relu, out=out, owner=m, name="weight")
                x = At(t, m.weight.shape[0], H, W)
                continue
            x = At(net.pack(N.PACK), Cc, H, W)
        pool = mods[i] if i < len(mods) and isinstance(mods[i], nn.MaxPool2d) and not net.nchw else None
        if pool is not None:
            i += 1
            out = planes_next(i)
        x = conv(net, m, x, scale, shift, relu, precision, out=out, pool=pool)
    if x is None:
        raise NotExpressible
    return classify(net, x, model.head.fc)


def build_densenet(model, net, precision):
    from .densenet import TKDenseBlock, TKDenseLayer, TKDenseNet, TKDenseTransition
    if type(model).forward_features is not TKDenseNet.forward_features:
        raise NotExpressible
    _average_to_one(model.global_pool)
    for name, m in model.features.named_children():
        if name.startswith(("denseblock", "transition")) and type(_exact(m, TKDenseBlock, TKDenseTransition)) is TKDenseBlock:
            for layer in m.values():
                _exact(layer, TKDenseLayer)
    if net.nchw:
        return build_densenet_nchw(model, net, precision)
    f = model.features
    B = net.shape[0]
    s, b, _ = fold_bn(f.norm0)
    x = stem7(net, f.conv0, s, b, f.pool0, N.PLANES, precision)
    stages = [m for name, m in f.named_children() if name.startswith(("denseblock", "transition"))]
    buf = None
    H = W = None
    for m in stages:
        if isinstance(m, TKDenseBlock):
            layers = list(m.values())
            if buf is None:
                Hs, Ws = net.shape[2], net.shape[3]
                H, W = _pooled(f.pool0, -(-Hs // 2)), _pooled(f.pool0, -(-Ws // 2))
            else:
                H, W = H // 2, W // 2
            if H <= 0 or W <= 0:
                raise NotExpressible
            buf = net.planes(B, m.num_output_features, H, W)
            x(into=buf)                                   # the block's input: its first channels
            c = m.num_input_features
            for layer in layers:
                s1, b1, bound1 = fold_bn(layer.norm1)
                s2, b2, _ = fold_bn(layer.norm2)
                a = At(net.pool(buf, 1, 1, out=N.PACKED, scale=s1, shift=b1, bound=bound1, channels=c), c, H, W)
                z = conv(net, layer.conv1, a, s2, b2, True, precision)
                conv(net, layer.conv2, z, None, None, False, precision, out=N.PLANES, into=buf, into_c=c)
                c += layer.growth_rate
        elif isinstance(m, TKDenseTransition):
            p = m.pool
            if (p.kernel_size, p.stride, p.padding) != (2, 2, 0) or p.ceil_mode or H < 2 or W < 2:
                raise NotExpressible
            s1, b1, bound1 = fold_bn(m.norm)
            # the average and the 1x1 convolution commute: averaging first leaves a quarter of the positions to convolve
            a = At(net.pool(buf, 2, 2, out=N.PACKED, scale=s1, shift=b1, bound=bound1), m.norm.num_features, H // 2, W // 2)
            x = (lambda cv, src: lambda into: conv(net, cv, src, None, None, False, precision, out=N.PLANES, into=into))(m.conv, a)
        else:
            raise NotExpressible
    if buf is None:
        raise NotExpressible
    s, b, _ = fold_bn(f.norm5)
    return classify(net, At(buf, f.norm5.num_features, H, W), model.classifier, s, b)


def build_densenet_nchw(model, net, precision):
    """The steps of TKDenseNet.forward, layer by layer: one feature buffer per block, new features copied into it."""
    from .densenet import TKDenseBlock, TKDenseTransition
    f = model.features
    s, b, _ = fold_bn(f.norm0)
    x = stem7(net, f.conv0, s, b, f.pool0, N.PLANES, precision)()
    for name, m in f.named_children():
        if isinstance(m, TKDenseBlock):
            if x.C != m.num_input_features:
                raise NotExpressible
            buf = net.nchw_buffer(m.num_output_features, x.H, x.W)
            net.nchw_affine(x.id, into=buf)
            c = x.C
            for layer in m.values():
                s1, b1, _ = fold_bn(layer.norm1)
                s2, b2, _ = fold_bn(layer.norm2)
                a = At(net.nchw_affine(buf, s1, b1, True, channels=c), c, x.H, x.W)
                z = conv(net, layer.conv1, a, s2, b2, True, precision)
                if precision != "fp32" and type(layer.conv2).__name__ == "TKConv2dC_B200" and layer.conv2.fold_pays():
                    # (as the layer-by-layer forward does: the last 1x1 step multiplied into the core filter)
                    k = layer.conv2
                    z = nchw_step(net, k, "first", z, k.first_kernel, None, None, False, precision, -1, 1, 0)
                    y = nchw_step(net, k, "core_last", z, k._core_last_weight(), None, _with_bias(k, None, None), False, precision, -1, k.stride[0], k.padding[0])
                else:
                    y = conv(net, layer.conv2, z, None, None, False, precision)
                net.nchw_affine(y.id, into=buf, into_c=c)
                c += y.C
            x = At(buf, c, x.H, x.W)
        elif isinstance(m, TKDenseTransition):
            p = m.pool
            if (p.kernel_size, p.stride, p.padding) != (2, 2, 0) or p.ceil_mode or x.H < 2 or x.W < 2:
                raise NotExpressible
            s1, b1, _ = fold_bn(m.norm)
            a = At(net.nchw_affine(x.id, s1, b1, True), x.C, x.H, x.W)
            z = conv(net, m.conv, a, None, None, False, precision)
            x = At(net.nchw_pool(z.id, 2, 2, 0, 1), z.C, z.H // 2, z.W // 2)      # average, padding included
        elif name.startswith(("denseblock", "transition")):
            raise NotExpressible
    s, b, _ = fold_bn(f.norm5)
    return classify(net, x, model.classifier, s, b)


def _pooled(m, n):
    k, s, p = ((v[0] if isinstance(v, (tuple, list)) else v) for v in (m.kernel_size, m.stride, m.padding))
    return (n + 2 * p - k) // s + 1


# ---- the cache on a model ----------------------------------------------------------------------------------------------
class Nets:
    """The nets of one model by input shape, and what they were built from: the modules and their classes, the tensors, the
    keys of every table of children, parameters and buffers, and the plain attributes the builders read."""
    READ = ("stride", "padding", "dilation", "groups", "kernel_size", "ceil_mode", "output_size", "eps", "in_channels", "out_channels", "in_rank", "out_rank", "rank",
            "num_features", "num_input_features", "num_output_features", "growth_rate", "in_features", "out_features", "downsample")
    MOST = 256                    # shapes kept, the oldest goes first: a net is 30 - 200 KB of host memory (filters live on the modules)

    def __init__(self, model=None, head=None):
        self.nets, self.lock = {}, threading.Lock()
        self.classifier = None                                # of the nets that run it themselves
        self.parts, self.tensors, self.modules, self.mark = [], [], [], None
        self.orders, self.sizes, self.lengths, self.read, self.values = [], [], [], [], []
        if model is not None:
            apart = set(head.modules())                       # called, or compared by its tensors' addresses (native_classifier)
            self.modules = [m for m in model.modules() if m not in apart and m is not model]      # (not the model itself: it holds this object)
            for m in [model] + self.modules:
                self.parts += [(m._modules, k, c) for k, c in m._modules.items()]
                for d in (m._parameters, m._buffers):
                    self.parts += [(d, k, None) for k, t in d.items() if t is None]
                    self.tensors += [(d, k) for k, t in d.items() if t is not None and t.dtype.is_floating_point]
                if m._modules:
                    self.orders.append((m._modules, list(m._modules)))
                self.sizes += [m._modules, m._parameters, m._buffers]
                self.read += [(m.__dict__, k) for k in self.READ if k in m.__dict__]
            self.lengths = [len(d) for d in self.sizes]
            self.values = [d[k] for d, k in self.read]
            self.blocks = [m for m in self.modules if "precision" in m.__dict__]
            self.types = [type(m) for m in [model] + self.modules]
            self.mark = self.state()

    def __deepcopy__(self, memo):
        return Nets()

    def __reduce__(self):
        return (Nets, ())

    def state(self):
        return [(t._version, t.data_ptr()) for t in [d.get(k) for d, k in self.tensors]]

    def plain(self, model):
        """Whether the submodules' own forwards would do what the network says: no hooks, eval mode, one precision, no forward of
        one object's own."""
        if _module._global_forward_hooks or _module._global_forward_pre_hooks or "forward_features" in model.__dict__:
            return False
        for m in self.modules:
            d = m.__dict__
            if m._forward_hooks or m._forward_pre_hooks or m.training or "forward" in d or "new_features" in d:
                return False
        return all(m.precision == model.precision for m in self.blocks)

    def current(self, model):
        """Whether the model still is what the nets were built from."""
        try:
            return self.mark is not None and all(d.get(k) is c for d, k, c in self.parts) and self.types == [type(m) for m in [model] + self.modules] \
                and self.lengths == [len(d) for d in self.sizes] and all(list(d) == keys for d, keys in self.orders) \
                and self.values == [d.get(k) for d, k in self.read] and self.state() == self.mark
        except AttributeError:        # a tensor is gone
            return False


def forward(model, x, build, head):
    """The model's output for x through its net, or None where it has to run layer by layer.  `head`: its classifier."""
    native = native_classifier(head, x)
    for _ in range(4):                # (found out of date, built, run)
        cache = model.__dict__.get("_nets")
        if cache is None or cache.mark is None or (native and cache.classifier not in (None, native)):
            cache = model.__dict__["_nets"] = Nets(model, head)
        key = (x.shape, x.device.index, model.precision, native is None)
        net = cache.nets.get(key)
        y = net(x) if net else None
        if not cache.current(model):
            model.__dict__["_nets"] = None
        elif net or net is False or not cache.plain(model):
            if y is None or not cache.plain(model):
                return None
            return y if native else head(y)
        else:
            with cache.lock:
                if key not in cache.nets:
                    with N.building(x.device):
                        built = _build(model, x, build, head, native is None)
                    N.make_room(cache.nets, Nets.MOST)
                    cache.classifier = native or cache.classifier
                    cache.nets[key] = built
    return None


def _build(model, x, build, head, features):
    try:
        apart = {id(p) for p in head.parameters()}
        if any(p.device != x.device or p.dtype != torch.float32 for p in model.parameters() if id(p) not in apart):
            return False
        net = N.Net(*x.shape, x.device)
        net.nchw, net.features = model.precision in NCHW_PRECISIONS, features
        return build(model, net, model.precision)
    except (NotExpressible, AttributeError, TypeError, IndexError, KeyError):      # (a module without what the builders read: the layers decide)
        return False
    except TdcError as e:
        if e.code in (ERR_SMEM, ERR_UNSUPPORTED, ERR_SHAPE):
            return False
        raise


# ---- one Tucker module -------------------------------------------------------------------------------------------------
class _LayerNet:
    """A module's nets by input shape, precision and device, and the factors they were built from."""
    MOST = 1024                   # (a few KB each)

    def __init__(self):
        self.nets, self.mark = {}, None

    def __deepcopy__(self, memo):
        return _LayerNet()

    def __reduce__(self):
        return (_LayerNet, ())


def layer(module, x):
    """A Tucker module's output for a contiguous fp32 x through its net, or None where it has to run step by step."""
    d = module.__dict__
    p = d["_parameters"]
    first, core, last, bias = p.get("first_kernel"), p.get("core_kernel"), p.get("last_kernel"), p.get("bias")
    if first is None or core is None or last is None:      # parametrised or pruned: they are made anew on every access
        return None
    mark = (first._version, first.data_ptr(), core._version, core.data_ptr(), last._version, last.data_ptr(),
            None if bias is None else (bias._version, bias.data_ptr()), d["stride"], d["padding"], d["dilation"], d["groups"])
    cache = d.get("_layer_net")
    if cache is None or cache.mark != mark:
        cache = d["_layer_net"] = _LayerNet()
        cache.mark = mark
        cache.keep = [t.detach() for t in (first, core, last, bias) if t is not None]      # the mark holds their addresses
    key = (x.shape, module.precision, x.device.index)
    net = cache.nets.get(key)
    if net is None:
        with N.building(x.device):
            net = _build_layer(module, x)
        N.make_room(cache.nets, _LayerNet.MOST)
        cache.nets[key] = net
    if not net:
        return None
    # (from module to module, and from and to TcConv, the exact range: only the first of a chain looks at its input)
    xmax = range_of(x) if "_tdc_absmax" in x.__dict__ else None
    if not net.leaves_range:
        return net(x, None, xmax)
    ymax = x.new_empty(ABSMAX_FLOATS)
    y = net(x, None, xmax, ymax)
    y._tdc_absmax = ymax
    return y


def _one_launch_wins(module, x):
    """A Tucker module on its own reads and writes NCHW: on large feature maps the packing pass costs more than the packed
    form saves, and the launches that split and gather as they go (dispatch.one_conv) are the faster way."""
    from . import dispatch as D
    B, Cc, H, W = x.shape
    K, R1, R2 = module.out_channels, module.in_rank, module.out_rank
    dense = _estimate(B, Cc, H, W, False, N.CONV3x3, K, False, N.NCHW)
    chain = _estimate(B, Cc, H, W, False, N.CONV1x1, R1, False, N.PACKED) + _estimate(B, R1, H, W, False, N.CONV3x3, R2, False, N.PACKED) \
        + _estimate(B, R2, H, W, False, N.CONV1x1, K, False, N.NCHW)
    packed = D.packed_us(B, Cc, K, H, W, H, W, min(dense, chain))
    if D.tucker_strategy(module, x, "auto") == "dense":
        direct = D.one_launch_us(B, Cc, K, H, W, 3, 1)
    else:
        direct = D.one_launch_us(B, Cc, R1, H, W, 1, 1) + D.one_launch_us(B, R1, R2, H, W, 3, 1) + D.one_launch_us(B, R2, K, H, W, 1, 1)
    return direct <= max(13.3, packed)          # (the host time of a call that packs: TcConv._packs)


def _began_in_fp32(module, x):
    """Whether the layer-by-layer form of a module under "auto" begins in fp32 arithmetic, which takes any input: on packed operands that
    wants the true maximum.  (Where it begins on tensor cores it samples, and so does packing.)"""
    from . import dispatch as D
    B, Cc, H, W = x.shape
    if D.tucker_strategy(module, x, "auto") == "dense":
        return not D._on_tensor_cores(B, Cc, module.out_channels, H, W, 3, 3, module.stride[0], 1)
    return not D._on_tensor_cores(B, Cc, module.in_rank, H, W, 1, 1, 1, 0)


def _ended_in_fp32(module, x, Ho, Wo):
    """Likewise its end, which then leaves no range; small calls are over sooner than the table for one is allocated."""
    from . import dispatch as D
    B, Cc, H, W = x.shape
    if D.tucker_strategy(module, x, "auto") == "dense":
        return _began_in_fp32(module, x)
    return not D._on_tensor_cores(B, module.out_rank, module.out_channels, Ho, Wo, 1, 1, 1, 0)


def _build_layer(module, x):
    from . import dispatch, tc
    try:
        if any(t is not None and (t.device != x.device or t.dtype != torch.float32) for t in module._parameters.values()):
            return False
        B, Cc, H, W = x.shape
        if Cc != module.in_channels:
            return False
        if module.precision in NCHW_PRECISIONS:
            # the three steps on the kernels of dispatch.one_conv, made from native code (three calls from Python cost 40 us of
            # host time, one 11)
            net, bias = N.Net(B, Cc, H, W, x.device), None if module.bias is None else module.bias.detach()
            z = nchw_step(net, module, "first", At(-1, Cc, H, W), module.first_kernel, None, None, False, module.precision, -1, 1, 0)
            z = nchw_step(net, module, "core", z, module.core_kernel, None, None, False, module.precision, -1, module.stride[0], module.padding[0])
            z = nchw_step(net, module, "last", z, module.last_kernel, None, bias, False, module.precision, -1, 1, 0, to_y=True)
            return net.finish((B, z.C, z.H, z.W))
        stride = _square(module, 3)
        net = N.Net(B, Cc, H, W, x.device)
        K, shape = module.out_channels, (B, module.out_channels, -(-H // stride), -(-W // stride))
        auto = module.precision == "auto"
        if not (auto and stride == 1 and _one_launch_wins(module, x)):
            at = At(net.pack(N.PACK_SPLIT if stride == 2 else N.PACK, auto and _began_in_fp32(module, x)), Cc, H, W, stride == 2)
            conv(net, module, at, None, None, False, module.precision, out=N.NCHW)
            net.leaves_range = not (auto and _ended_in_fp32(module, x, *shape[2:]))
            return net.finish(shape)

        # the launches of the layer-by-layer path (dispatch.one_conv under "auto"), made from native code
        def step(src, name, w, last=False):
            k, c, R = w.shape[:3]
            plan, flt, flags = None, None, 0
            if tc.supported(R, R, 1, R // 2, W) and dispatch._on_tensor_cores(B, c, k, H, W, R, R, 1, R // 2) and not dispatch._thin_and_wide(c, W, R, 1):
                plan, flt, flags = tc.cached(module, name, w, dispatch.AUTO_MODE).step(B, H, W, 1, None)
            else:
                flt = dispatch.channel_last(module, name, w)
            bias = module.bias.detach() if last and module.bias is not None else None
            return net.nchw_conv(src, k, R, 1, R // 2, flt, None, bias, -1, False, plan, flags, to_y=last)
        if dispatch.tucker_strategy(module, x, "auto") == "dense":
            step(-1, "dense", module._dense_weight(), True)
        else:
            step(step(step(-1, "first", module.first_kernel), "core", module.core_kernel), "last", module.last_kernel, True)
        return net.finish(shape)
    except NotExpressible:
        return False
    except TdcError as e:
        if e.code in (ERR_SMEM, ERR_UNSUPPORTED, ERR_SHAPE):
            return False
        raise
