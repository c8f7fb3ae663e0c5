"""Which networks run as a net of prepared launches, and when a net is made anew: the builders and the cache of programs.py
on the CPU, with a stand-in for the library's object that records the steps."""
import types

import pytest
import torch
import torch.nn as nn


class Steps:
    """Takes the calls of net.Net and keeps them; running it gives zeros of the output's shape."""
    made = []

    def __init__(self, B, C, H, W, device):
        self.shape, self.device, self.nchw, self.features, self.steps = (B, C, H, W), device, False, False, []
        Steps.made.append(self)

    def _step(self, *what):
        self.steps.append(what)
        return len(self.steps)

    def pack(self, kind=0):
        return self._step("pack", kind)

    def conv(self, src, kind, weight, **kw):
        return self._step("conv", src, kind, tuple(weight.shape), kw.get("residual", -1))

    def planes(self, *shape):
        return self._step("planes", *shape)

    def pool(self, src, k, stride, pad=0, **kw):
        return self._step("pool", src, k, stride, pad)

    def head(self, src, weight=None, *a, **kw):
        return self._step("head" if weight is not None else "averages", src)

    def finish(self, out_shape):
        self.out_shape = tuple(out_shape)
        return self

    def __call__(self, x):
        return torch.zeros(self.out_shape)


@pytest.fixture
def P(built, monkeypatch):
    from tdc_b200 import programs
    Steps.made = []
    monkeypatch.setattr(programs.N, "Net", Steps)
    monkeypatch.setattr(programs, "_estimate", lambda *a, **kw: 1.0)
    monkeypatch.setattr(programs, "_pooled_estimates", lambda *a, **kw: (2.0, 1.0))
    monkeypatch.setattr(programs, "fold_bn", lambda bn: (bn.running_var, bn.running_mean, bn.running_var[:2]))
    return programs


def nets(T):
    return {"resnet18": (T.tkc_resnet18, "build_resnet", 64), "resnet50": (T.tkc_resnet50, "build_resnet", 64), "vgg": (lambda **k: T.TKVGG(cfg=[8, "M", 16], **k), "build_vgg", 16),
            "densenet": (lambda **k: T.TKDenseNet(8, (2, 2), num_classes=10, **k), "build_densenet", 64)}


def make(P, name, **kw):
    """(model, a call that gives its net's output or None where it has to run layer by layer)"""
    import tdc_b200 as T
    from tdc_b200 import densenet, vgg  # noqa: F401
    T = types.SimpleNamespace(tkc_resnet18=T.tkc_resnet18, tkc_resnet50=T.tkc_resnet50, TKVGG=vgg.TKVGG, TKDenseNet=densenet.TKDenseNet)
    ctor, build, size = nets(T)[name]
    model = ctor(precision="auto", **kw).eval()

    def call(B=1, H=size, W=size, channels=3, grad=False):
        with torch.set_grad_enabled(grad):
            return P.forward(model, torch.zeros(B, channels, H, W), getattr(P, build), model.get_submodule(HEADS[name]))
    return model, call


HEADS = {"resnet18": "fc", "resnet50": "fc", "vgg": "head.fc", "densenet": "classifier"}


NAMES = ("resnet18", "resnet50", "vgg", "densenet")


@pytest.mark.parametrize("name", NAMES)
def test_the_stock_networks_are_nets(P, name):
    model, call = make(P, name)
    assert call() is not None and len(Steps.made) == 1
    assert call() is not None and len(Steps.made) == 1


class Scaled(nn.Linear):
    def forward(self, x):
        return 2 * super().forward(x)


def with_own_forward(block):
    class Own(block):
        def forward(self, x):
            return 2 * super().forward(x)
    return Own


REPLACED = {
    "avgpool": ("resnet18", lambda m: setattr(m, "avgpool", nn.AdaptiveMaxPool2d(1))),
    "maxpool": ("resnet18", lambda m: setattr(m, "maxpool", nn.AvgPool2d(2))),
    "avgpool's size": ("resnet18", lambda m: setattr(m, "avgpool", nn.AdaptiveAvgPool2d(2))),
    "stage": ("resnet18", lambda m: setattr(m, "layer4", nn.Identity())),
    "stage with its own forward": ("resnet50", lambda m: setattr(m.layer2, "__class__", type("S", (nn.Sequential,), {"forward": lambda self, x: x}))),
    "block with its own forward": ("resnet18", lambda m: setattr(m.layer1[0], "__class__", with_own_forward(type(m.layer1[0])))),
    "bottleneck with its own forward": ("resnet50", lambda m: setattr(m.layer1[0], "__class__", with_own_forward(type(m.layer1[0])))),
    "a forward of one block": ("resnet18", lambda m: setattr(m.layer1[0], "forward", lambda x: x)),
    "global_pool": ("densenet", lambda m: setattr(m, "global_pool", nn.AdaptiveMaxPool2d(1))),
    "dense block with its own forward": ("densenet", lambda m: setattr(m.features.denseblock1, "__class__", with_own_forward(type(m.features.denseblock1)))),
    "transition with its own forward": ("densenet", lambda m: setattr(m.features.transition1, "__class__", with_own_forward(type(m.features.transition1)))),
    "dense layer of another kind": ("densenet", lambda m: setattr(m.features.denseblock1.denselayer1, "__class__",
                                                                 type("L", (type(m.features.denseblock1.denselayer1),), {"new_features": lambda self, p, q: p}))),
    "new features of one layer": ("densenet", lambda m: setattr(m.features.denseblock1.denselayer1, "new_features", lambda p, q: p)),
    "features of a subclass": ("densenet", lambda m: setattr(m, "__class__", type("D", (type(m),), {"forward_features": lambda self, x: x}))),
    "features of a VGG subclass": ("vgg", lambda m: setattr(m, "__class__", type("V", (type(m),), {"forward_features": lambda self, x: x}))),
}


@pytest.mark.parametrize("what", sorted(REPLACED))
@pytest.mark.parametrize("before", [True, False])
def test_a_module_that_does_something_else_is_called(P, what, before):
    """What the layer-by-layer forward calls — stages, blocks, the average pool — a net may only replace where it is the module
    whose arithmetic the net has; replaced before the first call and after it."""
    name, change = REPLACED[what]
    model, call = make(P, name)
    if not before:
        assert call() is not None
    change(model)
    assert call() is None and call() is None


@pytest.mark.parametrize("name", sorted(HEADS))
@pytest.mark.parametrize("head", ["identity", "chain", "subclass"])
@pytest.mark.parametrize("before", [True, False])
def test_any_classifier_is_called(P, name, head, before):
    """The launch of a net stands for nn.Linear; another module is called on the averages."""
    model, call = make(P, name)
    if not before:
        assert call() is not None and Steps.made[-1].steps[-1][0] == "head"
    owner, _, leaf = HEADS[name].rpartition(".")
    n = model.get_submodule(HEADS[name]).in_features
    own = {"identity": nn.Identity, "chain": lambda: nn.Sequential(nn.Linear(n, 7)), "subclass": lambda: Scaled(n, 7)}[head]().eval()
    setattr(model.get_submodule(owner), leaf, own)
    y = call()
    assert torch.equal(y, own(torch.zeros(1, n))) and Steps.made[-1].steps[-1][0] == "averages"


def called(P, monkeypatch, name="resnet18"):
    """(model, call, the list of the inputs its classifier was called on)"""
    model, call = make(P, name)
    seen, forward = [], nn.Linear.forward
    monkeypatch.setattr(nn.Linear, "forward", lambda self, x: seen.append(x.shape) or forward(self, x))
    return model, call, seen


def test_the_classifier_has_its_gradient(P, monkeypatch):
    """A frozen network whose classifier is trained: with gradients enabled the classifier is torch's, without them the net's."""
    model, call, seen = called(P, monkeypatch)
    y = call(grad=True)
    y.sum().backward()
    assert seen == [(1, 512)] and model.fc.weight.grad is not None and torch.equal(model.fc.bias.grad, torch.ones(1000))
    assert not call().requires_grad and len(seen) == 1
    model.fc.requires_grad_(False)
    assert not call(grad=True).requires_grad and len(seen) == 1


def test_what_torch_does_around_a_call_reaches_the_classifier(P, monkeypatch):
    """Autocast, forward-mode derivatives, function transforms, dispatch modes and hooks on the classifier."""
    from torch.utils._python_dispatch import TorchDispatchMode
    model, call, seen = called(P, monkeypatch)
    assert call() is not None and not seen
    with torch.autocast("cpu", dtype=torch.bfloat16):
        assert call().dtype == torch.bfloat16 and len(seen) == 1
    with torch.autograd.forward_ad.dual_level():
        assert call() is not None and len(seen) == 2
    torch.func.vmap(lambda v: v + call().sum())(torch.zeros(2))
    assert len(seen) == 3

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))
    with Mode():
        assert call() is not None and len(seen) == 4
    h = model.fc.register_forward_hook(lambda *a: None)
    assert call() is not None and len(seen) == 5
    h.remove()
    model.fc.train()
    assert call() is not None and len(seen) == 5


def test_a_replaced_classifier_weight_is_read(P):
    """A net's last launch reads the weight where it lies: written in place it counts at once, replaced it means another net."""
    model, call = make(P, "resnet18")
    call()
    with torch.no_grad():
        model.fc.weight.mul_(2)
    call()
    assert len(Steps.made) == 1
    model.fc.weight = nn.Parameter(torch.zeros(5, 512))
    model.fc.bias = None
    assert call().shape == (1, 5) and len(Steps.made) == 2


def test_hooks_on_every_module(P):
    """torch.nn.modules.module.register_module_forward_hook: every module has to be called."""
    model, call = make(P, "resnet18")
    assert call() is not None
    h = nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert call() is None
    finally:
        h.remove()
    assert call() is not None


def appended_block(m):
    import tdc_b200.resnet as R
    m.layer1.append(R.TKBasicBlock(64, 64, stage=1, id=1, hp_dict=R.HalfRanks()).eval())
    m.layer1[-1].precision = m.precision


CHANGED = {
    "appended block": ("resnet18", appended_block),
    "order of the children": ("resnet18", lambda m: m.layer1._modules.move_to_end("0") if hasattr(m.layer1._modules, "move_to_end")
                              else m.layer1._modules.__setitem__("0", m.layer1._modules.pop("0"))),
    "a new child": ("vgg", lambda m: m.features.add_module("9", nn.MaxPool2d(2).eval())),
    "eps": ("resnet50", lambda m: setattr(m.layer3[0].bn2, "eps", 0.5)),
    "pool geometry": ("resnet18", lambda m: setattr(m.maxpool, "kernel_size", 5) or setattr(m.maxpool, "padding", 2)),
    "stride of a convolution": ("resnet18", lambda m: setattr(m.layer2[0].conv1, "stride", (1, 1)) or setattr(m.layer2[0].downsample[0], "stride", (1, 1))),
    "a shortcut taken out": ("resnet18", lambda m: setattr(m.layer1[0], "downsample", None) or setattr(m.layer1[1], "downsample", nn.Sequential(nn.Conv2d(64, 64, 1), nn.BatchNorm2d(64)).eval())),
    "a bias": ("densenet", lambda m: m.features.conv0.register_parameter("bias", nn.Parameter(torch.zeros(16)))),
    "a weight": ("vgg", lambda m: m.features[0].weight.mul_(2)),
}


@pytest.mark.parametrize("what", sorted(CHANGED))
def test_what_a_net_was_built_from_is_compared(P, what):
    """Structure, plain attributes and tensors: each of these changes what the layer-by-layer forward computes."""
    name, change = CHANGED[what]
    model, call = make(P, name)
    assert call() is not None and call() is not None and len(Steps.made) == 1
    with torch.no_grad():
        change(model)
    call()
    assert len(Steps.made) == 2
    call()
    assert len(Steps.made) == 2


def test_a_network_that_becomes_expressible_is_a_net_again(P):
    model, call = make(P, "resnet18")
    pool, model.avgpool = model.avgpool, nn.AdaptiveMaxPool2d(1)
    assert call() is None and call() is None
    model.avgpool = pool
    assert call() is not None


def test_folded_batchnorm_notices_eps(built, monkeypatch):
    """The fold is kept on the module until one of its tensors, or eps, changes."""
    from tdc_b200 import programs
    asked = []
    monkeypatch.setattr(programs, "lib", types.SimpleNamespace(tdc_net_fold_bn=lambda *a: asked.append(a[4]) or 0))
    monkeypatch.setattr(programs, "_stream", lambda: 0)
    bn = nn.BatchNorm2d(8).eval()
    programs.fold_bn(bn), programs.fold_bn(bn)
    bn.eps = 0.25
    programs.fold_bn(bn)
    assert asked == [1e-5, 0.25]


def test_tucker_module_notices_its_geometry(built, monkeypatch):
    """A Tucker module's net is for one stride and padding."""
    import tdc_b200 as T
    from tdc_b200 import programs

    class HP:
        ranks = {"l": [8, 8]}
    made = []
    monkeypatch.setattr(programs, "_build_layer", lambda m, x: made.append((m.stride, m.padding)) or False)
    m = T.TKConv2dC_B200(16, 16, 3, padding=1, hp_dict=HP, name="l")
    x = torch.zeros(1, 16, 8, 8)
    for stride, padding in (((1, 1), (1, 1)), ((1, 1), (1, 1)), ((2, 2), (1, 1)), ((2, 2), (0, 0))):
        m.stride, m.padding = stride, padding
        assert programs.layer(m, x) is None
    assert made == [((1, 1), (1, 1)), ((2, 2), (1, 1)), ((2, 2), (0, 0))]


@pytest.mark.parametrize("name,channels", [("resnet18", 1), ("vgg", 1), ("vgg", 4), ("vgg", 20), ("densenet", 1)])
def test_input_of_other_channels_is_left_to_the_layers(P, name, channels):
    """(whose checks refuse it)"""
    model, call = make(P, name)
    assert call(channels=channels) is None


def test_filters_and_vectors_match_their_tensor(built):
    """The launches read the sizes of the tensor behind the pointers of filter, scale, bias and classifier: a mismatch is refused
    before the library is asked."""
    from tdc_b200 import TdcError, net as N
    n = object.__new__(N.Net)
    n._h, n._keep, n._channels, n.clocks, n.shape = None, [], {-1: 16, 0: 16}, 0.0, (1, 16, 8, 8)
    ok, w = torch.zeros(8), torch.zeros(8, 16, 1, 1)
    for call in (lambda: n.conv(0, N.CONV1x1, torch.zeros(8, 17, 1, 1)), lambda: n.conv(0, N.CONV3x3_ROWS, torch.zeros(8, 16, 3, 3)), lambda: n.conv(0, N.CONV7x7_S2, torch.zeros(8, 5, 7, 7)),
                 lambda: n.conv(1, N.CONV1x1, w), lambda: n.conv(0, N.CONV1x1, w, torch.zeros(7), ok), lambda: n.conv(0, N.CONV1x1, w, ok, torch.zeros(9)),
                 lambda: n.pool(0, 1, 1, scale=ok, shift=ok, bound=ok), lambda: n.pool(0, 1, 1, scale=ok, shift=ok, bound=ok, channels=4),
                 lambda: n.nchw_conv(-1, 8, 1, 1, 0, w, scale=torch.zeros(16)), lambda: n.nchw_affine(-1, ok, ok), lambda: n.head(0, torch.zeros(10, 17), None),
                 lambda: n.head(0, torch.zeros(10, 16), torch.zeros(9))):
        with pytest.raises(TdcError) as e:
            call()
        assert e.value.code == 2          # TDC_ERR_SHAPE


def test_bias_and_batchnorm_are_folded_once(built):
    """What a net's launches read lives on the modules: a net that makes room for another shape's takes nothing with it that a graph
    captured from it still reads."""
    from tdc_b200 import programs
    conv, scale, shift = nn.Conv2d(4, 8, 1), torch.rand(8) + 0.5, torch.rand(8)
    first = programs._with_bias(conv, scale, shift)
    assert torch.equal(first, shift + conv.bias.detach() * scale) and programs._with_bias(conv, scale, shift) is first
    with torch.no_grad():
        conv.bias.add_(1)
    again = programs._with_bias(conv, scale, shift)
    assert again is not first and torch.equal(again, shift + conv.bias.detach() * scale)
    shift.mul_(2)
    assert torch.equal(programs._with_bias(conv, scale, shift), shift + conv.bias.detach() * scale)
    assert programs._with_bias(conv, None, None).data_ptr() == conv.bias.data_ptr()


def test_rotating_shapes_stay_built(P):
    """Forty input sizes in turn: each is built once.  The table is bounded all the same, and threads may make room at once."""
    import threading
    from tdc_b200 import net as N
    model, call = make(P, "vgg")
    for _ in range(2):
        for i in range(40):
            assert call(H=16 + i) is not None
    assert len(Steps.made) == 40
    for i in range(P.Nets.MOST):
        call(H=100 + i)
    assert len(model._nets.nets) == P.Nets.MOST
    table, wrong = {i: i for i in range(500)}, []

    def work(k):
        try:
            for i in range(2000):
                N.make_room(table, 400)
                table[(k, i)] = 1
        except Exception as e:      # noqa: BLE001
            wrong.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong and len(table) <= 408


def test_parametrised_factors_run_step_by_step(built):
    """A parametrised or pruned factor is no parameter of the module any more, and is made anew on every access."""
    import tdc_b200 as T
    from tdc_b200 import programs

    class HP:
        ranks = {"l": [8, 8]}
    m = T.TKConv2dC_B200(16, 16, 3, padding=1, hp_dict=HP, name="l")
    nn.utils.parametrize.register_parametrization(m, "first_kernel", nn.Identity())
    assert programs.layer(m, torch.zeros(1, 16, 8, 8)) is None


def test_range_of_a_tensor_ends_when_it_is_written_to():
    from tdc_b200 import ops
    y, bound = torch.zeros(4), torch.ones(8)
    assert ops.range_of(y) is None
    ops.leave_range(y, bound)
    assert ops.range_of(y) is bound
    y.view(2, 2).add_(1)
    assert ops.range_of(y) is None
    with torch.inference_mode():          # (no version to compare)
        z = torch.zeros(4)
        ops.leave_range(z, bound)
        assert ops.range_of(z) is bound


def test_copies_start_without_what_is_kept_by_address(built, monkeypatch):
    """A copied or loaded module's tensors may lie where the original's did, with the same version."""
    import copy
    import pickle
    from tdc_b200 import dispatch, net, programs
    monkeypatch.setattr(programs, "lib", types.SimpleNamespace(tdc_net_fold_bn=lambda *a: 0))
    monkeypatch.setattr(net, "lib", types.SimpleNamespace(tdc_net_filter_prepare=lambda *a: 0))
    monkeypatch.setattr(dispatch.ops, "permute_weights", lambda w: w.permute(1, 2, 3, 0).contiguous())
    monkeypatch.setattr(net, "_dev_f32", lambda t, name: t.data_ptr())
    for m in (programs, net):
        monkeypatch.setattr(m, "_stream", lambda: 0)
    conv, bn = nn.Conv2d(4, 8, 1), nn.BatchNorm2d(8).eval()
    programs.fold_bn(bn)
    programs._with_bias(conv, torch.rand(8), torch.rand(8))
    dispatch.channel_last(conv, "weight", conv.weight)
    net.Net._filter(None, net.CONV1x1, conv.weight, 32, 64, None, None, conv, "weight")
    kept = {"_tdc_fold": bn, "_tdc_shift": conv, "_channel_last": conv, "_net_filters": conv}
    assert all(m.__dict__[name] for name, m in kept.items())
    for again in (copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))):
        assert not any(again(m).__dict__[name] for name, m in kept.items())


@pytest.mark.parametrize("what", ["double", "strided", "no affine"])
def test_folded_batchnorm_of_other_types_and_layouts(built, monkeypatch, what):
    """The library's fold reads fp32 values that lie next to each other; statistics of another type or layout are not handed to it."""
    from tdc_b200 import programs
    monkeypatch.setattr(programs, "lib", types.SimpleNamespace(tdc_net_fold_bn=lambda *a: pytest.fail("called")))
    bn = nn.BatchNorm2d(8, affine=what != "no affine").eval()
    bn.running_var, bn.running_mean = torch.rand(8).double() + 0.5, torch.randn(8).double()
    if what == "strided":
        bn.running_var, bn.running_mean = (torch.rand(8, 3) + 0.5)[:, 1], torch.randn(8)
    scale, shift, bound = programs.fold_bn(bn)
    g, b = (1.0, 0.0) if bn.weight is None else (bn.weight.detach().double(), bn.bias.detach().double())
    s = g / (bn.running_var.double() + bn.eps).sqrt()
    assert torch.equal(scale, s.float()) and torch.equal(shift, (b - bn.running_mean.double() * s).float())
    assert bound.tolist() == [float(scale.abs().max()), float(shift.abs().max())]
