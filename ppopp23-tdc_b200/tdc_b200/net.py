"""Chains of convolutions on packed activations (tdc_net_* of the C ABI): what the networks and the large tensor-core layers
run on under fp16 parts.

`Net` is the thin wrapper: it numbers tensors, prepares filters (kept on the module that owns the weight, one per kind,
block size and epilogue) and holds everything the built object points to.  A net is built for one input shape and keeps the
identity of every tensor it was built from (`fresh` says whether they are still the ones): weights written to or replaced
mean another build."""
import ctypes as C
import threading

import torch

from . import _lib
from ._lib import ERR_SHAPE, NetConv, NetNchw, NetPool, TdcError, check, lib
from .ops import _dev_f32, _on_device, _stream

PACK, PACK_SPLIT, PACK_S2D, PACK_ROWS = range(4)
PACK_EXACT = 0x100
CONV1x1, CONV3x3, CONV3x3_S2, CONV7x7_S2, CONV3x3_ROWS, CONV1x1_S2 = range(6)
PACKED, PLANES, NCHW = 1, 2, 4


def _key(*tensors):
    return tuple((t._version, t.data_ptr()) if t is not None else None for t in tensors)


# ---- work that is done once and read on any stream --------------------------------------------------------------------------
def _mark(device):
    """An event behind what the current stream was given so far (None under capture: a replay repeats the work in place)."""
    if device.index is None or torch.cuda.is_current_stream_capturing():
        return None
    event = torch.cuda.Event()
    event.record()
    return event


class building:
    """`with building(device):` around work whose results are kept — prepared filters, folded BatchNorms, channel-last copies.  They
    are shared between nets, and the next net may be built by another thread on another stream: one is built at a time,
    and its stream first waits for the work of the one before."""
    _lock, _depth, _nets, _made = threading.RLock(), 0, [], False
    _last = {}          # device -> (the event behind the last such work, the stream it was put on)

    def __init__(self, device):
        self.device, self.on = device, _on_device(device)

    def __enter__(self):
        building._lock.acquire()
        building._depth += 1
        self.on.__enter__()
        if building._depth > 1:
            building._made = True
            return
        building._made = False
        last = building._last.get(self.device.index)
        if last is not None and last[1] != _stream() and not torch.cuda.is_current_stream_capturing():
            torch.cuda.current_stream().wait_event(last[0])

    def __exit__(self, *exc):
        try:
            if building._depth == 1:
                if building._made:
                    event = _mark(self.device)
                    if event is not None:
                        building._last[self.device.index] = (event, _stream())
                for net in building._nets:
                    net._event, net._built_on = building._last.get(self.device.index, (None, None))
                building._nets.clear()
        finally:
            building._depth -= 1
            self.on.__exit__(*exc)
            building._lock.release()

    @staticmethod
    def made():
        """Says that something was prepared (without it a build leaves no event: it only read what was there)."""
        building._made = True


def make_room(table, most):
    """Drops the oldest entries until one more fits (another thread may be at the same table)."""
    while len(table) >= most:
        try:
            table.pop(next(iter(table)), None)
        except (StopIteration, RuntimeError):
            pass


class Cache(dict):
    """Nets and prepared memory kept on an object that may be copied or pickled.  A net is a handle to memory of this process, and what
    is kept under the addresses of tensors says nothing about another object's or process's: a copy starts without them."""

    def __deepcopy__(self, memo):
        return Cache()

    def __reduce__(self):
        return (Cache, ())


class Net:
    def __init__(self, B, Cc, H, W, device):
        self.device = device
        self.shape = (B, Cc, H, W)
        self._h = C.c_void_p()
        self._keep = []                 # everything the launches point to
        self._channels = {-1: Cc}       # tensor -> its channels (-1: the input)
        self._event, self._built_on, self._streams = None, None, set()
        self.leaves_range = False       # a run writes the partial maxima of |y| it is given room for
        self.nchw, self.features = False, False      # which steps the network builders take, and whether they end at the classifier (programs.py)
        self.clocks = 0.0
        with _on_device(device):
            check(lib.tdc_net_create(C.byref(self._h), B, Cc, H, W))

    def __del__(self):
        if getattr(self, "_h", None) and lib is not None:      # (module globals are gone at interpreter exit)
            lib.tdc_net_destroy(self._h)
            self._h = None

    def pack(self, kind=PACK, exact=False):
        """`exact`: the true maximum of an input of any size (of up to 2^18 values it is found anyway)."""
        out = C.c_int()
        check(lib.tdc_net_pack(self._h, kind | (PACK_EXACT if exact else 0), C.byref(out)))
        return self._made(out.value, self.shape[1] * {PACK_S2D: 4, PACK_ROWS: 3}.get(kind, 1))

    def _made(self, tensor, channels):
        self._channels[tensor] = channels
        return tensor

    @staticmethod
    def _per_channel(channels, *vectors):
        """The launches read one value per channel behind these pointers."""
        for v in vectors:
            if v is not None and v.numel() != channels:
                raise TdcError(ERR_SHAPE, "%d values for %d channels" % (v.numel(), channels))

    def conv(self, src, kind, weight, scale=None, bias=None, relu=False, residual=-1, out=PACKED, split=False, into=-1, into_c=0,
             owner=None, name=None, unbiased=True, tile=None, pool=0):
        """`weight`: [K][C][R][R] tensor.  With an `owner` module the prepared filter is kept there under `name`."""
        K, Cc = weight.shape[:2]
        # (the prepared filter's size follows from the tensor, its contents from the weight)
        if Cc * {CONV7x7_S2: 4, CONV3x3_ROWS: 3}.get(kind, 1) != self._channels.get(src, -1):
            raise TdcError(ERR_SHAPE, "a filter of %d channels on tensor %d of %s" % (Cc, src, self._channels.get(src)))
        self._per_channel(K, scale, bias)
        d = NetConv()
        d.kind, d.K, d.relu, d.residual, d.out, d.out_split, d.into, d.into_c, d.unbiased = kind, K, int(relu), residual, out, int(split), into, into_c, int(unbiased)
        d.pool = pool
        d.scale = _dev_f32(scale, "scale") if scale is not None else None
        d.bias = _dev_f32(bias, "bias") if bias is not None else None
        if tile is not None:
            d.nt, d.mt, d.ks = tile
        check(lib.tdc_net_conv_plan(self._h, src, C.byref(d)))
        self.clocks += d.clocks
        self.leaves_range |= out == NCHW
        flt = self._filter(kind, weight, d.nt, d.filter_bytes, scale, bias, owner, name)
        d.filter = flt.data_ptr()
        self._keep += [flt, scale, bias]
        t = C.c_int()
        check(lib.tdc_net_add_conv(self._h, src, C.byref(d), C.byref(t)))
        return t.value if into >= 0 or out == NCHW else self._made(t.value, K)

    def _filter(self, kind, weight, nt, nbytes, scale, bias, owner, name):
        store = owner.__dict__.setdefault("_net_filters", Cache()) if owner is not None else {}
        at, key = (name, kind, nt, scale is None, bias is None), _key(weight, scale, bias)
        hit = store.get(at)
        if hit is None or hit[0] != key:
            building.made()
            w = weight.detach()
            buf = torch.empty(nbytes, dtype=torch.uint8, device=w.device)
            check(lib.tdc_net_filter_prepare(kind, w.shape[0], w.shape[1], nt, _dev_f32(w, "weight"), scale.data_ptr() if scale is not None else None,
                                             bias.data_ptr() if bias is not None else None, buf.data_ptr(), _stream()))
            # (the key holds addresses: the memory they belong to stays alive with it, whatever becomes of the parameter)
            hit = store[at] = (key, buf, w, scale, bias)
        return hit[1]

    def planes(self, B, Cc, H, W):
        t = C.c_int()
        check(lib.tdc_net_planes(self._h, B, Cc, H, W, C.byref(t)))
        return self._made(t.value, Cc)

    def pool(self, src, k, stride, pad=0, out=PACKED, scale=None, shift=None, bound=None, channels=0, into=-1):
        channels_out = channels or self._channels.get(src, -1)
        self._per_channel(channels_out, scale, shift)
        d = NetPool()
        d.k, d.stride, d.pad, d.channels, d.out, d.into = k, stride, pad, channels, out, into
        for n, t in (("scale", scale), ("shift", shift), ("bound", bound)):
            setattr(d, n, _dev_f32(t, n) if t is not None else None)
        self._keep += [scale, shift, bound]
        t = C.c_int()
        check(lib.tdc_net_pool(self._h, src, C.byref(d), C.byref(t)))
        return t.value if into >= 0 else self._made(t.value, channels_out)

    # -- NCHW steps (source -1: the input) ----------------------------------------------------------------------------
    def nchw_conv(self, src, K, R, stride, pad, flt, scale=None, bias=None, residual=-1, relu=False, plan=None, flags=0, to_y=False):
        self._per_channel(K, scale, bias)
        d = NetNchw()
        d.K, d.R, d.S, d.stride, d.pad, d.flags, d.residual, d.relu = K, R, R, stride, pad, flags, residual, int(relu)
        d.to_y = int(to_y)
        self.leaves_range |= bool(to_y) and plan is not None and plan.mode == 4
        d.plan = C.pointer(plan) if plan is not None else None
        d.filter = flt.data_ptr()
        d.scale = _dev_f32(scale, "scale") if scale is not None else None
        d.bias = _dev_f32(bias, "bias") if bias is not None else None
        self._keep += [flt, scale, bias]
        t = C.c_int()
        check(lib.tdc_net_nchw_conv(self._h, src, C.byref(d), C.byref(t)))
        return t.value if to_y else self._made(t.value, K)

    def nchw_pool(self, src, k, stride, pad, mode):
        t = C.c_int()
        check(lib.tdc_net_nchw_pool(self._h, src, k, stride, pad, mode, C.byref(t)))
        return self._made(t.value, self._channels.get(src, -1))

    def nchw_buffer(self, Cc, H, W):
        t = C.c_int()
        check(lib.tdc_net_nchw_buffer(self._h, Cc, H, W, C.byref(t)))
        return self._made(t.value, Cc)

    def nchw_affine(self, src, scale=None, shift=None, relu=False, channels=0, into=-1, into_c=0):
        channels_out = channels or self._channels.get(src, -1)
        self._per_channel(channels_out, scale, shift)
        self._keep += [scale, shift]
        t = C.c_int()
        check(lib.tdc_net_nchw_affine(self._h, src, channels, scale.data_ptr() if scale is not None else None, shift.data_ptr() if shift is not None else None,
                                      int(relu), into, into_c, C.byref(t)))
        return t.value if into >= 0 else self._made(t.value, channels_out)

    def head(self, src, weight=None, bias=None, scale=None, shift=None):
        """Global average and classifier; without a weight the averages alone."""
        self._per_channel(self._channels.get(src, -1), scale, shift)
        w = b = None
        if weight is not None:
            weight, bias = weight.detach(), bias.detach() if bias is not None else None      # (aliases: the launches read this memory)
            self._per_channel(self._channels.get(src, -1), weight[0])
            self._per_channel(weight.shape[0], bias)
            w, b = _dev_f32(weight, "weight"), _dev_f32(bias, "bias") if bias is not None else None
        self._keep += [weight, bias, scale, shift]
        check(lib.tdc_net_head(self._h, src, scale.data_ptr() if scale is not None else None, shift.data_ptr() if shift is not None else None,
                               w, b, weight.shape[0] if weight is not None else 0))

    def finish(self, out_shape):
        n = C.c_size_t()
        check(lib.tdc_net_finish(self._h, C.byref(n)))
        self.arena_bytes, self.out_shape = n.value, tuple(out_shape)
        self.arena_floats = max(1, -(-n.value // 4))
        if building._lock._is_owned():
            building._nets.append(self)             # (its event: the end of the build, before anyone is handed the net)
        else:
            self._event = _mark(self.device)
        return self

    def meet(self, stream):
        """Before the first run on a stream: the run waits for what was prepared for the net, wherever that was, and the memory it
        reads is not given to anyone else while the stream may still be reading it, whatever becomes of the net."""
        if torch.cuda.is_current_stream_capturing():      # (captures begin on an idle device; what a graph reads is for its owner to keep)
            return
        current = torch.cuda.current_stream()
        if self._event is not None and stream != self._built_on:
            current.wait_event(self._event)
        for t in self._keep:
            if t is not None and t.is_cuda:
                t.record_stream(current)
        self._streams.add(stream)

    def __call__(self, x, out=None, x_absmax=None, y_absmax=None, factors=None):
        """`factors`: (scale, bias) of this run, either may be None, in place of those the last convolution was built with."""
        if out is None:
            out = x.new_empty(self.out_shape)
        arena = x.new_empty(self.arena_floats)
        if factors is None and self.device.index == torch.cuda.current_device():
            # (the lean form of the call below: a batch-1 layer is over in less time than the interpreter's detours take)
            stream = _stream()
            if stream not in self._streams:
                self.meet(stream)
            code = lib.tdc_net_run(self._h, x.data_ptr(), None if x_absmax is None else x_absmax.data_ptr(), out.data_ptr(),
                                   None if y_absmax is None else y_absmax.data_ptr(), arena.data_ptr(), self.arena_bytes, stream)
            if code:
                check(code)
            return out
        with _on_device(x.device):
            stream = _stream()
            if stream not in self._streams:
                self.meet(stream)
            xm, ym = (t.data_ptr() if t is not None else None for t in (x_absmax, y_absmax))
            if factors is None:
                check(lib.tdc_net_run(self._h, x.data_ptr(), xm, out.data_ptr(), ym, arena.data_ptr(), self.arena_bytes, stream))
            else:
                s, b = (_dev_f32(t, "scale or bias") if t is not None else None for t in factors)
                check(lib.tdc_net_run_scaled(self._h, x.data_ptr(), xm, s, b, out.data_ptr(), ym, arena.data_ptr(), self.arena_bytes, stream))
        return out
