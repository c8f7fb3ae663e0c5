"""Tensor-core variant of the core convolution (tcgen05, TF32 or fp16 operands) — host side.

`TcConv` holds what the C ABI needs per layer: the plan (tdc_tc_plan_make) and the filter
pre-arranged for the kernel (tdc_tc_prepare_weights).  mode 3 ("3xTF32") and mode 4 ("3xFP16")
give fp32-level results; mode 1 is plain TF32.  Mode 4 scales its input into fp16's range and needs
the input's largest magnitude for that: every mode-4 output carries the partial maxima of its own
magnitudes as the attribute `_tdc_absmax`, and a mode-4 call whose input carries one skips the pass
over the input that would otherwise find it (the three steps of a Tucker conv chain this way).  The default plan serves "same" convolutions with 1x1 or 3x3 filters
and stride 1 (1x1 filters also strided) and reads the input once; `general=True` makes the plan that
takes any filter size, stride and padding by gathering (channel, row, column) triples.
"""
import ctypes as C
import os

import torch

from . import _lib
from ._lib import TcPlan, TdcError, lib
from .net import Cache, building, make_room
from .ops import ABSMAX_FLOATS, _dev_f32, _epilogue, _on_device, _stream, leave_range, range_of


def _check(code):
    if code != _lib.OK:
        raise TdcError(code, lib.tdc_tc_last_error_string().decode())


# the tuning switches are those of the one-launch kernels: with TDC_TC_TUNING set they are what runs
_TUNING = os.environ.get("TDC_TC_TUNING", "0") not in ("", "0")


class TcConv:
    # mode 4: a pass that packs the input for the tensor cores and a convolution on packed activations (net.py) instead of the
    # one launch that splits and gathers as it goes.  None: where it is the faster of the two (`_packs`)
    packed = None

    def __init__(self, weight, mode=3, w_layout=_lib.W_KCRS, general=False, exact_range=False, unbiased=False, snapshot=True):
        """weight: [K][C][R][S] (or [C][R][S][K] with w_layout=W_CRSK), fp32 CUDA tensor.  `exact_range` (mode 4): take
        the input's scale from its true maximum (a pass over the input per call) instead of from a sample.  `unbiased`
        (modes 3, 4): put back the expected loss of the tensor core's truncating accumulation (TDC_TC_UNBIASED); sums of
        small integers are then no longer exact.  `snapshot`: the layer is that of `weight` as it is now; further forms of it (other
        block sizes, packed) are prepared from a copy when a shape first needs them.  False: from `weight` itself, which the
        owner then does not write to while the layer is used."""
        self.exact_range, self.unbiased = bool(exact_range), bool(unbiased)
        if w_layout == _lib.W_KCRS:
            K, Cc, R, S = weight.shape
        else:
            Cc, R, S, K = weight.shape
        self.plan = TcPlan()
        _check((lib.tdc_tc_plan_make_general if general else lib.tdc_tc_plan_make)(Cc, K, R, S, mode, C.byref(self.plan)))
        self.C, self.K, self.R, self.S, self.mode, self.general = Cc, K, R, S, mode, bool(general)
        self._weight, self._w_layout = weight, w_layout
        self._by_nt = {(self.plan.nt, None): (self.plan, self._prepare(self.plan))}   # (output-channel block size, strided-row (stride, padding parity)) -> (plan, prepared filter)
        if snapshot:
            self._weight = weight.detach().clone()
        self._nets = Cache()                                     # (input shape, stride, padding, ReLU, switches) -> net on packed activations, or None
        self._plain = Cache()                                    # (input shape, stride, padding) -> what a plain call on it launches
        self._sms = torch.cuda.get_device_properties(weight.device).multi_processor_count
        self._nt_of = {}                                         # (batch, image, flags) -> block size (the rules are library calls)

    def _prepare(self, plan):
        wt = torch.empty(plan.weights_bytes, dtype=torch.uint8, device=self._weight.device)
        with torch.cuda.device(self._weight.device):
            _check(lib.tdc_tc_prepare_weights(C.byref(plan), _dev_f32(self._weight, "weight"), self._w_layout,
                                              wt.data_ptr(), _stream()))
        return wt

    def _make_plan(self, nt, rows):
        plan = TcPlan()
        if rows:
            _check(lib.tdc_tc_plan_make_strided(self.C, self.K, self.R, self.S, rows[0], rows[1], self.mode, nt, C.byref(plan)))
        else:
            _check(lib.tdc_tc_plan_make_nt(self.C, self.K, self.R, self.S, self.mode, int(self.general), nt, C.byref(plan)))
        return plan

    def _for_image(self, B, H, W, Ho, Wo, flags, rows=None):
        """(plan, prepared filter) with the output-channel block size that suits this layer: the default for layers with
        many position tiles, smaller blocks (more CTAs) for few, and smaller again while the block does not leave room
        for two stages beside the patch of a wide image; prepared on first use.  `rows` = (stride, parity of the padding):
        the strided-row plan for them instead of the triple-gathering one."""
        halo = 0 if self.general else (self.R - 1) // 2
        key = (B, H, W, flags, rows)
        nt = self._nt_of.get(key)
        if nt is None:
            nt = lib.tdc_tc_pick_nt(self.K, self.mode, B * (Ho + halo) * (Wo + halo), self._sms)
            while nt > 32:
                plan = self._make_plan(nt, rows)
                if lib.tdc_tc_check_launch(C.byref(plan), B, H, W, flags & 0xFF) != _lib.ERR_SMEM:
                    break
                nt //= 2
            self._nt_of[key] = nt
        hit = self._by_nt.get((nt, rows))
        if hit is None:
            plan = self._make_plan(nt, rows)
            hit = self._by_nt[(nt, rows)] = (plan, self._prepare(plan))
        return hit

    MOST = 1024          # shapes kept, the oldest goes first

    def _remember(self, asked, rec):
        make_room(self._plain, self.MOST)
        self._plain[asked] = rec

    def step(self, B, H, W, stride, padding):
        """(plan, prepared filter, flags) of a call on this shape, for a net that makes it (not the strided-row plan)."""
        if self.general:
            flags = (stride - 1) | padding << 4
            Ho, Wo = (H + 2 * padding - self.R) // stride + 1, (W + 2 * padding - self.S) // stride + 1
        else:
            flags = stride - 1
            Ho, Wo = (H - 1) // stride + 1, (W - 1) // stride + 1
        plan, wt = self._for_image(B, H, W, Ho, Wo, flags)
        return plan, wt, flags | (0x200 if self.unbiased and self.mode != 1 else 0)          # TDC_TC_UNBIASED

    def _net(self, x, relu, stride, padding):
        """The net that runs this call on packed activations, or None: another filter than 1x1, 3x3 or 7x7 / 2 in its "same"
        form, or a shape the one-launch kernel is faster on.  Scale and bias come with each run."""
        key = (x.shape, stride, padding, relu, self.unbiased, self.packed)
        hit = self._nets.get(key, self)
        if hit is self:
            make_room(self._nets, self.MOST)
            hit = self._nets[key] = self._make_net(x, relu, stride, padding)
        return hit

    def _make_net(self, x, relu, stride, padding):
        from . import net as N
        kind, pack = {(1, 1): (N.CONV1x1, N.PACK), (3, 1): (N.CONV3x3, N.PACK), (3, 2): (N.CONV3x3_S2, N.PACK_SPLIT), (1, 2): (N.CONV1x1_S2, N.PACK_SPLIT),
                      (7, 2): (N.CONV7x7_S2, N.PACK_S2D)}.get((self.R, stride), (None, None))
        B, Cc, H, W = x.shape
        if kind is None or self.R != self.S or (padding is not None and padding != self.R // 2):
            return None
        # (what the one launch refuses stays refused, by it)
        if not self.general and stride > 1 and self.R != 1:
            return None
        rows = (stride, padding & 1) if self.general and strided_rows(self.S, stride) else None
        plan = self._make_plan(self.plan.nt, rows) if rows else self.plan
        flags = (stride - 1) | (padding << 4 if self.general else 0)
        if lib.tdc_tc_check_launch(C.byref(plan), B, H, W, flags) in (_lib.ERR_UNSUPPORTED, _lib.ERR_SHAPE):
            return None
        if kind == N.CONV3x3 and 3 * Cc <= 16:
            kind, pack = N.CONV3x3_ROWS, N.PACK_ROWS
        if self.packed is None and (_TUNING or not self._packs(kind, B, Cc, H, W, stride)):
            return None
        w = self._weight if self._w_layout == _lib.W_KCRS else self._weight.permute(3, 0, 1, 2).contiguous()
        try:
            with N.building(x.device):
                net = N.Net(B, Cc, H, W, x.device)
                net.conv(net.pack(pack), kind, w, None, None, relu, out=N.NCHW, owner=self, name="weight", unbiased=self.unbiased)
                return net.finish((B, self.K, -(-H // stride), -(-W // stride)))
        except TdcError as e:
            if e.code in (_lib.ERR_SMEM, _lib.ERR_UNSUPPORTED, _lib.ERR_SHAPE):
                return None
            raise

    def _packs(self, kind, B, Cc, H, W, stride):
        """Whether the packed form is the faster one, by the estimates of both (dispatch.one_launch_us says where they come
        from).  The 7x7 / 2 form gains the fixed part of its loader (batch 1: 10 against 16 us) and loses a tenth on large
        batches (32 images: 65 against 60 us); three-channel 3x3 layers on wide images gain throughout (224x224, 32 images:
        201 against 350 us), and so does every 3x3 / 2 layer (33 of 7 - 112 pixels, batch 1 - 128: 1.1 - 15 times)."""
        from . import dispatch, net as N
        if self.R == 7:
            return B * H * W <= 8 * 224 * 224
        if kind == N.CONV3x3_ROWS:
            return W >= 64
        if kind == N.CONV3x3_S2:
            return True
        d = _lib.NetConv()
        d.kind, d.K, d.residual, d.out, d.into = kind, self.K, -1, N.NCHW, -1
        if lib.tdc_net_estimate(B, Cc, H, W, int(stride > 1), C.byref(d)) != _lib.OK:
            return False
        # (a call that is over sooner than the host can make the next costs its host time: 13.3 us with two launches and an
        # arena, 10.5 with one launch)
        return max(13.3, dispatch.packed_us(B, Cc, self.K, H, W, -(-H // stride), -(-W // stride), d.clocks)) < max(10.5, dispatch.one_launch_us(B, Cc, self.K, H, W, self.R, stride))

    def __call__(self, x, scale=None, bias=None, residual=None, relu=False, out=None, stride=1, padding=None):
        """`stride` > 1 is taken for 1x1 filters (the down-sampling shortcut of a residual stage) and by general
        plans, which also take any `padding` (the others pad (R-1)/2)."""
        # a shape this layer has run before, with nothing but the convolution asked for: no checks but those of the tensor,
        # and a third of the host time (a small layer is over sooner than the interpreter's way to its launch)
        rec = self._plain.get((x.shape, stride, padding)) if (scale is None and bias is None and residual is None and not relu and out is None) else None
        if rec is not None and rec[4] == x.device.index == torch.cuda.current_device() and x.dtype is torch.float32 and x.is_contiguous() and self.packed is None \
                and self.unbiased is rec[6] and not self.exact_range and not _TUNING:
            net, plan, wt, flags = rec[:4]
            if net is not None:
                ymax = x.new_empty(ABSMAX_FLOATS)
                out = x.new_empty(net.out_shape)
                xmax = range_of(x) if "_tdc_absmax" in x.__dict__ else None
                arena = x.new_empty(net.arena_floats)
                stream = _stream()
                if stream not in net._streams:
                    net.meet(stream)
                code = lib.tdc_net_run(net._h, x.data_ptr(), xmax.data_ptr() if xmax is not None else None, out.data_ptr(), ymax.data_ptr(), arena.data_ptr(),
                                       net.arena_bytes, stream)
                if code:
                    _check(code)
                out._tdc_absmax = ymax
                return out
            B, _, H, W = x.shape
            out = x.new_empty(rec[5])
            if self.mode != 4:
                code = lib.tdc_conv2d_tc(plan, x.data_ptr(), wt.data_ptr(), out.data_ptr(), B, H, W, None, flags, _stream())
            else:
                ymax = x.new_empty(ABSMAX_FLOATS)
                xmax = range_of(x) if "_tdc_absmax" in x.__dict__ else None
                code = lib.tdc_conv2d_tc_ranged(plan, x.data_ptr(), wt.data_ptr(), out.data_ptr(), B, H, W, None, flags,
                                                xmax.data_ptr() if xmax is not None else None, ymax.data_ptr(), _stream())
                out._tdc_absmax = ymax
            if code:
                _check(code)
            return out
        B, Cc, H, W = x.shape
        if Cc != self.C:
            raise TdcError(_lib.ERR_SHAPE, "x has %d channels, the filter expects %d" % (Cc, self.C))
        if not 1 <= stride <= 16:
            raise TdcError(_lib.ERR_UNSUPPORTED, "stride %d" % stride)
        flags = stride - 1
        asked, plain = (x.shape, stride, padding), scale is None and bias is None and residual is None and not relu and out is None and not self.exact_range
        if self.general:
            padding = 0 if padding is None else padding
            if not 0 <= padding <= 15:
                raise TdcError(_lib.ERR_UNSUPPORTED, "padding %d" % padding)
            flags |= padding << 4
            Ho, Wo = (H + 2 * padding - self.R) // stride + 1, (W + 2 * padding - self.S) // stride + 1
        else:
            if padding is not None and padding != (self.R - 1) // 2:
                raise TdcError(_lib.ERR_UNSUPPORTED, "this plan pads (R-1)/2; make it with general=True for padding %d" % padding)
            Ho, Wo = (H - 1) // stride + 1, (W - 1) // stride + 1
        if self.mode == 4 and residual is None and not self.exact_range and self.packed is not False:
            _dev_f32(x, "x")
            net = self._net(x, bool(relu), stride, padding)
            if net is not None:
                if out is None:
                    out = torch.empty(net.out_shape, device=x.device, dtype=torch.float32)
                else:
                    _dev_f32(out, "out")
                ymax = torch.empty(ABSMAX_FLOATS, device=x.device, dtype=torch.float32)
                net(x, out, range_of(x), ymax, None if scale is None and bias is None else (scale, bias))
                leave_range(out, ymax)
                if plain:
                    self._remember(asked, (net, None, None, 0, x.device.index, net.out_shape, self.unbiased))
                return out
        if out is None:
            out = torch.empty((B, self.K, Ho, Wo), device=x.device, dtype=torch.float32)
        e = _epilogue(scale, bias, residual, relu)
        # strided filters 2 or 4 strides wide (the 3x3 stride-2 cores, the 7x7 stride-2 stem): the strided-row plan, whose
        # loaders gather C*R*stride values per position instead of C*R*S
        rows = (stride, padding & 1) if (self.general and self.mode == 4 and strided_rows(self.S, stride)) else None
        plan, wt = self._for_image(B, H, W, Ho, Wo, flags, rows)
        if self.unbiased and self.mode != 1:
            flags |= 0x200                        # TDC_TC_UNBIASED
        if plain:
            self._remember(asked, (None, C.byref(plan), wt, flags, x.device.index, (B, self.K, Ho, Wo), self.unbiased))
        if self.mode != 4:
            with _on_device(x.device):
                _check(lib.tdc_conv2d_tc(C.byref(plan), _dev_f32(x, "x"), wt.data_ptr(), _dev_f32(out, "out"),
                                         B, H, W, C.byref(e), flags, _stream()))
            return out
        xmax = range_of(x)
        if xmax is None and self.exact_range:
            flags |= 0x100                        # TDC_TC_EXACT_RANGE
        ymax = torch.empty(ABSMAX_FLOATS, device=x.device, dtype=torch.float32)
        with _on_device(x.device):
            _check(lib.tdc_conv2d_tc_ranged(C.byref(plan), _dev_f32(x, "x"), wt.data_ptr(), _dev_f32(out, "out"),
                                            B, H, W, C.byref(e), flags, xmax.data_ptr() if xmax is not None else None,
                                            ymax.data_ptr(), _stream()))
        leave_range(out, ymax)
        return out


def supported(R, S, stride, padding, W):
    """True when the tensor-core variant is built for this convolution."""
    return R == S and R in (1, 3) and (stride == 1 or (R == 1 and 1 <= stride <= 16)) and padding == (R - 1) // 2 and W <= 256 * stride


def general_supported(R, S, stride, padding, Wo):
    """True when a general plan (any filter, stride, padding) can run this convolution."""
    return 1 <= R <= 15 and 1 <= S <= 15 and 1 <= stride <= 16 and 0 <= padding <= 15 and Wo <= 256


def strided_rows(S, stride):
    """True when a strided convolution takes the plan that gathers (channel, filter row, column phase) and runs the
    column steps as 2 or 4 MMA taps (fp16 parts only): 3-wide to 8-wide filters at stride 2, for instance."""
    return stride >= 2 and -(-S // stride) in (2, 4)


def worthwhile(B, C, H, W, K, R):
    """The tensor-core kernel works on tiles of 128 positions x up to 128 channels; with too few position tiles or too
    little arithmetic the fp32 kernel with its channel slices and clusters is the faster one.  The thresholds are a fit
    to 420 layers (3x3 and 1x1, 32..2048 channels, 7..56 pixels, batch 1..64) timed on both paths in one run
    (tests/golden/tc_vs_fp32_times_b200.json, which a CPU test holds the rule to).  A 3x3
    layer wants 3 position tiles and 0.1 GFLOP: 0.2 % from always taking the faster path.  A 1x1 layer with few tiles
    is one CTA walking all input channels, about 12 us + 0.085 us per channel whatever the tile count, while the fp32
    kernel's time follows the arithmetic; the three cases below are 1.2 % from the faster path (the thresholds they
    replace, which asked for 12..24 tiles: 4.3 %), and on CUDA-graphed forwards at batch 1..16 they are never slower
    and up to 23 % faster (TK-ResNet-50 at batch 4: 2.50 -> 1.91 ms; TK-DenseNet-121 at batch 8: 4.70 -> 3.65 ms)."""
    pad = (R - 1) // 2
    flops, positions = 2.0 * B * H * W * C * K * R * R, B * (H + pad) * (W + pad)
    if R == 1:
        tiles = positions / 128.0
        return (tiles >= 4 and flops >= 0.02e9) or (C <= 512 and flops >= 0.2e9) or \
               (tiles >= 3 and K >= 2 * C and flops >= 0.1e9)
    return flops >= 0.1e9 and positions >= 3 * 128


def cached(owner, name, weight, mode, w_layout=_lib.W_KCRS, general=False):
    """TcConv for `weight`, kept on the module that owns the weight (`owner`) under `name`, and
    rebuilt when the tensor is written to or replaced (version / storage check).  Keeping it on the
    owner — not in a table keyed by address — means a freed network's entries can never be taken
    for those of a new network whose weights happen to land on the same addresses.  These are the convolutions of the
    modules and networks, which chain many layers: they run with `unbiased` set."""
    store = owner.__dict__.setdefault("_tc_convs", {})
    key = (weight._version, weight.data_ptr(), tuple(weight.shape))
    hit = store.get((name, mode, w_layout, general))
    if hit is None or hit[0] != key:
        with building(weight.device):
            building.made()
            hit = store[(name, mode, w_layout, general)] = (key, TcConv(weight.detach(), mode, w_layout, general, unbiased=True, snapshot=False))
    return hit[1]


def status():
    """Device status word of the tensor-core kernels (synchronises): 0 = no bounded wait ran out."""
    s = C.c_int(-1)
    _check(lib.tdc_tc_status(C.byref(s)))
    return s.value
