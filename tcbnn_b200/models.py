"""Network topologies of the reference drivers as data, seeded synthetic weights and inputs,
and the GPU runner that chains the layer objects.

A topology is a list of layer specs (dicts).  The same list drives the GPU runner here and the
CPU oracle runner used by the tests, so both sides execute the identical network.

Topologies follow the reference drivers, not the textbook networks:
  * resnet18   : imagenet_resnet.cu:223-325 -- 7x7 stride-4 first layer (56x56x64, residual
                 saved), 16 binary 3x3 convs in 8 basic blocks (64/128/256/512; stride 2 at the
                 start of stages 2-4), every second conv adds the previous block's integer
                 residual (2x2 max-pooled when the stage changes), FC 25088->512, out 512->1000.
  * resnet_cifar: cifar10_resnet.cu:189-259 -- three-stage variant on 32x32 images.
  * vgg_cifar  : cifar10_vgg.cu:162-199 -- conv 3->128, 128->128+pool, ->256, 256+pool, ->512,
                 512+pool (feeds FC), FC 8192->1024->1024, out ->10.
  * mlp        : mnist_mlp.cu:112-126 -- 784 -> 1024 -> 1024 -> 1024 -> 10.
  * alexnet, vgg16_imagenet : alexnet.cu:141-178, imagenet_vgg.cu:217-280 (11x11 / 5x5 filters,
                 192 / 384 channels, pooled layers at 224 x 224).
"""
import ctypes as C
import functools
import weakref

import numpy as np
import torch

from . import lib, ops, param


def resnet18_spec(batch, image=224, classes=1000):
    L = [dict(type="inconv", name="Conv1", H=image, W=image, R=7, S=7, C=3, O=64,
              stride=4, pool=1, save_residual=True)]

    def conv(name, C, O, stride=1, **kw):
        L.append(dict(type="conv", name=name, C=C, O=O, R=3, S=3, stride=stride, pool=1, **kw))

    # stage 1
    conv("L1B1C1", 64, 64)
    conv("L1B1C2", 64, 64, save_residual=True, inject=0, residual_channels=64)
    conv("L1B2C1", 64, 64)
    conv("L1B2C2", 64, 64, save_residual=True, inject=2, residual_channels=128)
    # stage 2
    conv("L2B1C1", 64, 128, stride=2)
    conv("L2B1C2", 128, 128, save_residual=True, inject=4, residual_channels=128, residual_pool=True)
    conv("L2B2C1", 128, 128)
    conv("L2B2C2", 128, 128, save_residual=True, inject=6, residual_channels=128)
    # stage 3
    conv("L3B1C1", 128, 256, stride=2)
    conv("L3B1C2", 256, 256, save_residual=True, inject=8, residual_channels=128, residual_pool=True)
    conv("L3B2C1", 256, 256)
    conv("L3B2C2", 256, 256, save_residual=True, inject=10, residual_channels=256)
    # stage 4
    conv("L4B1C1", 256, 512, stride=2)
    conv("L4B1C2", 512, 512, save_residual=True, inject=12, residual_channels=256, residual_pool=True)
    conv("L4B2C1", 512, 512)
    conv("L4B2C2", 512, 512, ahead_fc=True, inject=14, residual_channels=512)
    L.append(dict(type="fc", name="Fc1", N=512))
    L.append(dict(type="out", name="Fout", N=classes))
    return dict(name="resnet18", batch=batch, layers=L)


def resnet_cifar_spec(batch, image=32, classes=10):
    """cifar10_resnet.cu:189-259 -- 3x3 first layer to 128 channels (residual saved), three stages
    of two basic blocks (128/256/512, stride 2 at the start of stages 2 and 3), FC -> 512 -> out."""
    L = [dict(type="inconv", name="Conv1", H=image, W=image, R=3, S=3, C=3, O=128, stride=1, pool=1,
              save_residual=True)]

    def conv(name, C, O, stride=1, **kw):
        L.append(dict(type="conv", name=name, C=C, O=O, R=3, S=3, stride=stride, pool=1, **kw))

    conv("L1B1C1", 128, 128)
    conv("L1B1C2", 128, 128, save_residual=True, inject=0, residual_channels=128)
    conv("L1B2C1", 128, 128)
    conv("L1B2C2", 128, 128, save_residual=True, inject=2, residual_channels=128)
    conv("L2B1C1", 128, 256, stride=2)
    conv("L2B1C2", 256, 256, save_residual=True, inject=4, residual_channels=128, residual_pool=True)
    conv("L2B2C1", 256, 256)
    conv("L2B2C2", 256, 256, save_residual=True, inject=6, residual_channels=256)
    conv("L3B1C1", 256, 512, stride=2)
    conv("L3B1C2", 512, 512, save_residual=True, inject=8, residual_channels=256, residual_pool=True)
    conv("L3B2C1", 512, 512)
    conv("L3B2C2", 512, 512, ahead_fc=True, inject=10, residual_channels=512)
    L.append(dict(type="fc", name="Fc1", N=512))
    L.append(dict(type="out", name="Fout", N=classes))
    return dict(name="resnet_cifar", batch=batch, layers=L)


def vgg_cifar_spec(batch, image=32, classes=10):
    L = [dict(type="inconv", name="Conv1", H=image, W=image, R=3, S=3, C=3, O=128, stride=1, pool=1)]
    for name, C, O, pool, afc in [("Conv2", 128, 128, 2, False), ("Conv3", 128, 256, 1, False),
                                  ("Conv4", 256, 256, 2, False), ("Conv5", 256, 512, 1, False),
                                  ("Conv6", 512, 512, 2, True)]:
        L.append(dict(type="conv", name=name, C=C, O=O, R=3, S=3, stride=1, pool=pool, ahead_fc=afc))
    L += [dict(type="fc", name="Fc1", N=1024), dict(type="fc", name="Fc2", N=1024),
          dict(type="out", name="Fout", N=classes)]
    return dict(name="vgg_cifar", batch=batch, layers=L)


def alexnet_spec(batch, image=224, hidden=4096, classes=1000):
    """alexnet.cu:141-178 -- 11x11/4 first layer with 2x2 pool (64 channels), 5x5 64->192 with
    pool, 3x3 192->384, 384->256, 256->256 with pool (feeds FC), FC -> hidden -> hidden -> out."""
    L = [dict(type="inconv", name="Conv1", H=image, W=image, R=11, S=11, C=3, O=64, stride=4, pool=2),
         dict(type="conv", name="Conv2", C=64, O=192, R=5, S=5, stride=1, pool=2),
         dict(type="conv", name="Conv3", C=192, O=384, R=3, S=3, stride=1, pool=1),
         dict(type="conv", name="Conv4", C=384, O=256, R=3, S=3, stride=1, pool=1),
         dict(type="conv", name="Conv5", C=256, O=256, R=3, S=3, stride=1, pool=2, ahead_fc=True),
         dict(type="fc", name="Fc1", N=hidden), dict(type="fc", name="Fc2", N=hidden),
         dict(type="out", name="Fout", N=classes)]
    return dict(name="alexnet", batch=batch, layers=L)


def vgg16_imagenet_spec(batch, image=224, hidden=4096, classes=1000):
    """imagenet_vgg.cu:217-280 -- thirteen 3x3 layers (64, 64+pool, 128, 128+pool, 256, 256,
    256+pool, 512, 512, 512+pool, 512, 512, 512+pool feeding FC), FC -> hidden -> hidden -> out."""
    L = [dict(type="inconv", name="Conv1", H=image, W=image, R=3, S=3, C=3, O=64, stride=1, pool=1)]
    cfg = [(64, 64, 2), (64, 128, 1), (128, 128, 2), (128, 256, 1), (256, 256, 1), (256, 256, 2),
           (256, 512, 1), (512, 512, 1), (512, 512, 2), (512, 512, 1), (512, 512, 1), (512, 512, 2)]
    for i, (C, O, pool) in enumerate(cfg):
        L.append(dict(type="conv", name="Conv%d" % (i + 2), C=C, O=O, R=3, S=3, stride=1, pool=pool,
                      ahead_fc=(i == len(cfg) - 1)))
    L += [dict(type="fc", name="Fc1", N=hidden), dict(type="fc", name="Fc2", N=hidden),
          dict(type="out", name="Fout", N=classes)]
    return dict(name="vgg16_imagenet", batch=batch, layers=L)


def mlp_spec(batch, features=784, hidden=1024, classes=10):
    L = [dict(type="in", name="Fin", K=features),
         dict(type="fc", name="Fc1", N=hidden), dict(type="fc", name="Fc2", N=hidden),
         dict(type="fc", name="Fc3", N=hidden), dict(type="out", name="Fout", N=classes)]
    return dict(name="mlp", batch=batch, layers=L)


def layer_shapes(spec):
    """Resolve H/W/K of every layer by walking the chain; returns a list of dicts with the
    resolved fields added (H, W, OH, OW, K)."""
    out = []
    H = W = Cprev = K = None
    for l in spec["layers"]:
        l = dict(l)
        t = l["type"]
        if t == "in":
            K = l["K"]
        elif t in ("inconv", "conv"):
            if t == "inconv":
                H, W = l["H"], l["W"]
            else:
                l["H"], l["W"] = H, W
            s, p, R = l["stride"], l["pool"], l["R"]
            bh = (H + s - 1) // s
            bw = (W + s - 1) // s
            l["OH"], l["OW"] = (bh + p - 1) // p, (bw + p - 1) // p
            H, W, Cprev = l["OH"], l["OW"], l["O"]
            K = H * W * Cprev
        elif t in ("fc", "out"):
            l["K"] = K
            K = l["N"]
        out.append(l)
    return out


def synthetic_weights(spec, seed):
    """Arrays in launch_array order (utility.h:188-196): per conv layer filter[R*S][C][O] then
    thresholds[O]; per FC weight[K][N] then thresholds[N]; output layer weight, scale, bias.
    Weights are +-1 (Bernoulli 0.5), thresholds N(0, sqrt(fan_in)); the first layer's
    thresholds are scaled to its fp32 input range."""
    g = np.random.Generator(np.random.PCG64(seed))
    arrays = []

    def pm1(shape):
        return (g.integers(0, 2, size=shape, dtype=np.int8).astype(np.float32) * 2 - 1)

    for l in layer_shapes(spec):
        t = l["type"]
        if t == "inconv":
            arrays.append(pm1((l["R"] * l["S"], 3, l["O"])))
            arrays.append((g.standard_normal(l["O"]) * np.sqrt(3 * l["R"] * l["S"])).astype(np.float32))
        elif t == "conv":
            fan = l["C"] * l["R"] * l["S"]
            arrays.append(pm1((l["R"] * l["S"], l["C"], l["O"])))
            arrays.append((g.standard_normal(l["O"]) * np.sqrt(fan)).astype(np.float32))
        elif t == "fc":
            arrays.append(pm1((l["K"], l["N"])))
            arrays.append((g.standard_normal(l["N"]) * np.sqrt(l["K"])).astype(np.float32))
        elif t == "out":
            arrays.append(pm1((l["K"], l["N"])))
            arrays.append((g.standard_normal(l["N"]) * 0.1 + 1.0).astype(np.float32))
            arrays.append(g.standard_normal(l["N"]).astype(np.float32))
    return arrays


def synthetic_input(spec, seed, batch=None):
    """Seeded stand-in for the datasets, with the value ranges the reference readers produce:
    images are uint8 uniform, scaled to [0,1] and normalised per channel (data.cpp:295-315,
    534-542); MLP features are uniform[0,1) minus 0.5 because In128 binarises at 0."""
    g = np.random.Generator(np.random.PCG64(seed))
    B = batch or spec["batch"]
    first = spec["layers"][0]
    if first["type"] == "in":
        return (g.random((B, first["K"]), dtype=np.float32) - np.float32(0.5))
    u8 = g.integers(0, 256, size=(B, 3, first["H"], first["W"]), dtype=np.uint8)
    mean = np.array([0.485, 0.456, 0.406], dtype=np.float32).reshape(1, 3, 1, 1)
    std = np.array([0.229, 0.224, 0.225], dtype=np.float32).reshape(1, 3, 1, 1)
    return ((u8.astype(np.float32) / np.float32(255.0)) - mean) / std


# max |value| synthetic_input() can produce for images: (1 - 0.406) / 0.225
SYNTHETIC_IMAGE_ABS_BOUND = 2.65


def synthetic_input_u8(spec, seed, batch=None):
    """The same synthetic images as synthetic_input(), as bytes plus the per-channel table of
    their fp32 values: lut[c][v] is computed with the arithmetic synthetic_input() applies, so
    lut[c][u8] reproduces its output bit for bit.  Returns (uint8 [B][3][H][W], fp32 [3][256])."""
    g = np.random.Generator(np.random.PCG64(seed))
    B = batch or spec["batch"]
    first = spec["layers"][0]
    if first["type"] == "in":
        raise ValueError("byte input is for image networks")
    u8 = g.integers(0, 256, size=(B, 3, first["H"], first["W"]), dtype=np.uint8)
    mean = np.array([0.485, 0.456, 0.406], dtype=np.float32).reshape(3, 1)
    std = np.array([0.229, 0.224, 0.225], dtype=np.float32).reshape(3, 1)
    v = np.arange(256, dtype=np.float32).reshape(1, 256)
    lut = ((v / np.float32(255.0)) - mean) / std
    return u8, lut.astype(np.float32)


_FACTS = (torch.Tensor.data_ptr, torch.Tensor.size, torch.Tensor.stride)


def _input_facts(layers):
    t = layers[0].input_gpu
    return t.data_ptr(), t.size(), t.stride(), t.dtype, t.device


def _meet(some, others):
    """Whether an address range of one list overlaps one of the other."""
    for lo, hi in some:
        for start, end in others:
            if lo < end and start < hi:
                return True
    return False


@functools.lru_cache(maxsize=256)
def _one_launch_pays(widths, rows, settings, device):
    """tcbnn_fc_chain_pays, under the process-wide settings and on the device that it is asked for."""
    return lib.load().tcbnn_fc_chain_pays((C.c_int * len(widths))(*widths), len(widths) - 1, rows)


def _chain_pays(layers):
    """Whether an MLP's pass in one call is worth asking for: on so many rows, and faster than its layers' calls
    (tcbnn_fc_chain_pays, which takes 64 to 960 rows on 148 SMs: others are not asked about, 5 us in a first pass)."""
    first = layers[0]
    if type(first).__name__ != "In128LayerParam" or not 64 <= first.live <= 960 or len(layers) < 2:
        return False
    return _one_launch_pays(tuple([l.output_width for l in layers]), first.live, lib.settings_generation, torch._C._cuda_getDevice())


def _chain_call(layers):
    """The one call that makes an MLP's whole pass (tcbnn_fc_chain), or None where it does not apply: other
    layers, more rows or wider layers than it takes, inputs that are not the layer in front's outputs, or buffers that
    are not all apart (rows are not worked on at the same time)."""
    first, last = layers[0], layers[-1]
    if (type(first).__name__ != "In128LayerParam" or type(last).__name__ != "Out128LayerParam" or
            any(type(l).__name__ != "Fc128LayerParam" for l in layers[1:-1])):
        return None
    x, bits = first.input_gpu, first.output_gpu
    shape = first.live, first.input_width, bits.shape[1]
    keep, chain = [x, bits], (lib.ChainLayer * (len(layers) - 1))()
    for i, (prev, l) in enumerate(zip(layers, layers[1:])):
        a, w, out = l.input_gpu, l.weight_gpu, l.output_gpu
        p0, p1 = (l.bn_scale_gpu, l.bn_bias_gpu) if l is last else (l.bn_gpu, None)
        if (l.live != first.live or a.data_ptr() != prev.output_gpu.data_ptr() or a.shape[1] != prev.output_gpu.shape[1]
                or l.input_width != prev.output_width):
            return None
        ops._need_cuda(a, w, p0, p1)
        chain[i] = lib.ChainLayer(w.data_ptr(), w.shape[1], l.input_width, w.shape[0], p0.data_ptr(), p1.data_ptr() if p1 is not None else None,
                                  out.data_ptr(), out.shape[1])
        keep += [a, w, p0, p1, out]
    args = (ops._ptr(x), *shape, ops._ptr(bits), chain, len(chain))
    library = lib.load()
    if not library.tcbnn_fc_chain_fits(chain, len(chain), *shape) or not library.tcbnn_fc_chain_apart(*args):
        return None
    return "tcbnn_fc_chain", args, tuple(t for t in keep if t is not None)


def _pass_calls(layers):
    """[(entry point, arguments, what they point to)] of one pass, and whether it is one in which weights and parameters are
    complete once the first launch runs, which is when layers behind it may read or expand theirs: it begins
    with an input layer, and writes none of them itself (one layer's output as another's weight).  Otherwise the
    layers run as they do when called by themselves."""
    if layers[0].settles:
        chain = _chain_call(layers) if _chain_pays(layers) else None       # (its list costs the host 25 us)
        if chain:
            return [chain], True
        calls, ahead, written = [], [], []
        for l in layers:
            call = l._call_args(True)
            calls.append(call)
            l.memory(call[1], ahead, written)
        if not _meet(ahead, written):
            return calls, True
    return [l._call_args(False) for l in layers], False


class _Calls:
    """A network's layers' calls, prepared.  Once noted they serve while nothing but the input has changed of what
    they were prepared from: an attribute of a layer, its live batch, a descriptor, a process-wide
    setting (hold), the place or shape of a tensor (moved; t.data = ... changes these in place).

    A pass asks moved() behind its launches, under which the answer costs nothing (35 us for the 100 tensors
    of ResNet-18), and is made again if it has to be.  That is safe because the memory the calls point
    into is kept, the input's apart, which is compared in front, and harmless because every pass writes
    all that it reads."""

    noted = False

    def __init__(self, layers):
        device = layers[0].output_gpu.device
        while True:
            self.scratch = ops.shared_scratch(device)
            prepared, self.in_pass = _pass_calls(layers)
            if self.scratch is ops.shared_scratch(device):                   # (else replaced by a larger one on the way)
                break
        self.calls = [(lib.bound(name), args) for name, args, _ in prepared]
        self.chain = prepared[0][0] == "tcbnn_fc_chain"
        self.kept = [t for _, _, keep in prepared for t in keep if t is not layers[0].input_gpu]

    def note(self, layers):
        self.tensors = list({id(t): t for t in self.kept if torch.is_tensor(t)}.values())
        self.memory = [t.detach() for t in self.tensors]
        self.facts = [list(map(f, self.tensors)) for f in _FACTS]
        self.scratch = next((t for t in self.tensors if t is self.scratch), None)    # replaced when a larger layer asks for it
        self.descs = list({id(d): d for d in self.kept if isinstance(d, lib.ConvDesc)}.values())
        self.desc_facts = list(map(bytes, self.descs))
        self.layers = list(layers)
        self.states, self.changes = [l.state() for l in layers], param.changes
        self.settings, self.device = lib.settings_generation, torch._C._cuda_getDevice()
        self.noted = True

    def hold(self, layers):
        """Whether the layers would make the same calls now, whatever their input, if no tensor has moved."""
        if not self.noted or self.layers != layers:
            return False
        if self.changes != param.changes:
            if [l.state() for l in layers] != self.states:
                return False
            self.changes = param.changes
        return (list(map(bytes, self.descs)) == self.desc_facts and
                self.settings == lib.settings_generation and self.device == torch._C._cuda_getDevice() and
                (self.scratch is None or self.scratch is ops.shared_scratch(self.scratch.device)))

    def serves(self, x):
        """Whether the calls can be made on another input tensor as they are."""
        return not self.chain or bool(lib.load().tcbnn_fc_chain_apart(ops._ptr(x), *self.calls[0][1][1:]))

    def first(self, layers):
        """The first call, on the input that layers[0] now has."""
        if self.chain:
            f, args = self.calls[0]
            return f, (ops._ptr(layers[0].input_gpu), *args[1:])
        name, args, _ = layers[0]._call_args(self.in_pass)
        return lib.bound(name), args

    def moved(self):
        return any(list(map(f, self.tensors)) != g for f, g in zip(_FACTS, self.facts))


class _Pass:
    """_Calls on one input tensor, and the graph recorded of them."""

    def __init__(self, calls, layers, fresh=True):
        """fresh: the calls have just been prepared, on this input."""
        self.common, self.calls = calls, list(calls.calls)
        if not fresh:
            self.calls[0] = calls.first(layers)
        self.input = _input_facts(layers)
        self.seen, self.graph = 0, None

    def run(self):
        stream = ops._stream()
        for f, args in self.calls:
            if f(*args, stream) != 0:
                lib.check(1)

    def record(self):
        """The calls as a graph, or None where they cannot be recorded (another capture mode of the
        caller's, say): they then go on being made one by one."""
        graph = torch.cuda.CUDAGraph()
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                # thread_local: only this thread's calls are checked during the capture; another
                # thread (e.g. a communicator's watchdog polling its events) is left alone.  (Not
                # torch.cuda.graph: it collects garbage and empties the allocator's cache first, 50 to
                # 100 ms per graph, and the launches allocate nothing.)
                graph.capture_begin(capture_error_mode="thread_local")
                try:
                    self.run()
                finally:
                    graph.capture_end()
        except RuntimeError:
            return None
        return graph


class Network:
    """Chain of layer objects built from a spec, the way the reference drivers build theirs
    (new XLayerParam(...) ; initialize(config, prev->get_output_gpu(), residual))."""

    def __init__(self, spec, weights, input_host, input_abs_bound=None, input_lut=None, handover=True):
        """input_abs_bound: max |pixel value| the caller guarantees; with it the residual chain
        is provably small and is stored as int16 instead of int32.
        input_lut: images arrive as uint8 with this [3][256] table of their fp32 values.
        handover: producers write the pre-expanded input of the conv layers that follow them."""
        self.spec, self.live_batch = spec, None
        B = spec["batch"]
        cfg = weights if hasattr(weights, "read") else param.ArrayConfig(weights)
        self.layers = []
        prev = None
        for l in layer_shapes(spec):
            t = l["type"]
            if t == "in":
                obj = param.In128LayerParam(l["name"], B, l["K"]).initialize(input_host)
            elif t == "inconv":
                obj = param.InConv128LayerParam(l["name"], l["H"], l["W"], l["R"], l["S"], 3, l["O"], B,
                                                l["stride"], l["stride"], True, l["pool"], l["pool"],
                                                l.get("save_residual", False),
                                                input_abs_bound=input_abs_bound).initialize(
                                                    input_host, cfg, input_lut=input_lut)
            elif t == "conv":
                inj = l.get("inject")
                obj = param.Conv128LayerParam(l["name"], l["H"], l["W"], l["R"], l["S"], l["C"], l["O"], B,
                                              l["stride"], l["stride"], True, l["pool"], l["pool"],
                                              l.get("ahead_fc", False), l.get("save_residual", False),
                                              inj is not None, l.get("residual_channels", 0),
                                              l.get("residual_pool", False))
                res = self.layers[inj].get_output_residual_gpu() if inj is not None else None
                rb = self.layers[inj].residual_bound if inj is not None else None
                obj.initialize(cfg, prev.get_output_gpu(), res, rb)
            elif t == "fc":
                obj = param.Fc128LayerParam(l["name"], B, l["K"], l["N"]).initialize(cfg, prev.get_output_gpu())
            elif t == "out":
                obj = param.Out128LayerParam(l["name"], B, l["K"], l["N"]).initialize(cfg, prev.get_output_gpu())
            else:
                raise ValueError(t)
            self.layers.append(obj)
            prev = obj
        if handover:
            self._wire_handover()
            self._wire_units()
            self._wire_residual_layouts()

    def _wire_handover(self):
        """Consecutive conv layers: where the consumer runs on a pre-expanded input, its producer
        writes that input itself (tcbnn_conv_layer_x) and the consumer skips its expansion pass."""
        for prod, cons in zip(self.layers, self.layers[1:]):
            if type(cons).__name__ != "Conv128LayerParam":
                continue
            kind = type(prod).__name__
            if kind == "Conv128LayerParam":
                dense = prod.out_image_stride == prod.desc.OH * prod.desc.OW * ((prod.desc.O + 31) // 32)
                if not dense:
                    continue
            elif kind == "InConv128LayerParam":
                if getattr(prod, "specialized", None) is None:
                    continue
            else:
                continue
            planes = ops.new_planes(cons.desc, cons.input_gpu.device)
            if planes is None:
                continue
            prod.next_layer = (cons.desc, planes)
            cons.input_planes = planes
            if kind == "Conv128LayerParam" and prod.desc.pool != 1:
                cons.pooling_producer = prod

    def _wire_units(self):
        """FC layers on the tcgen05 GEMM: a producer that packs bits (the input layer, another FC layer) also
        writes them expanded, and where the network starts with an input layer, its launch expands the
        weights.  Both are done anew in every pass."""
        for prod, cons in zip(self.layers, self.layers[1:]):
            if type(cons).__name__ != "Fc128LayerParam":
                continue
            M, K, N, dev = cons.input_height, cons.input_width, cons.weight_width, cons.weight_gpu.device
            if type(prod).__name__ in ("In128LayerParam", "Fc128LayerParam"):
                cons.units_room = ops.fc_units(M, N, K, M, dev)
            if type(self.layers[0]).__name__ == "In128LayerParam":
                cons.weight_room = ops.fc_units(M, N, K, N, dev)
        self._use_units()

    def _use_units(self):
        """Expanded operands are written where the live batch has a layer's call on the kernel that reads them so:
        from 1024 to about 1190 rows, say, a layer of 1024 x 1024 reads packed rows whatever it is given."""
        expands = []
        for prod, cons in zip(self.layers, self.layers[1:]):
            if type(cons).__name__ != "Fc128LayerParam" or (cons.units_room is None and cons.weight_room is None):
                continue
            some = ops.fc_units_bytes(cons.live, cons.weight_width, cons.input_width, cons.live) > 0
            cons.reads_units = some and ops.gemm_route(
                ops.GEMM_BITS, cons.live, cons.input_gpu, cons.weight_gpu, cons.input_width, cons.workspace,
                cons.units_room is not None, cons.weight_room is not None) != ops.GEMM_ON_PACKED
            if cons.units_room is not None:
                cons.producer = weakref.ref(prod)         # (prod may hold cons: In128LayerParam.expands)
                cons.input_units = prod.next_units = cons.units_room if cons.reads_units else None
            cons.weight_units = cons.weight_room if some else None
            if cons.weight_units is not None and cons.reads_units:
                expands.append(cons)
        if type(self.layers[0]).__name__ == "In128LayerParam":
            self.layers[0].expands = tuple(expands)

    def _wire_residual_layouts(self):
        """An int16 residual tensor is kept in the chunk-major layout (TCBNN_RES_INT16_CHUNKED)
        when the layer that saves it and every layer that injects it move residual rows directly
        between registers and memory: one thread per pixel then touches whole lines per warp."""
        consumers = {}
        for l in self.layers:
            if type(l).__name__ == "Conv128LayerParam" and l.inject_residual:
                for p in self.layers:
                    if getattr(p, "output_residual_gpu", None) is l.input_residual_gpu and p.output_residual_gpu is not None:
                        consumers.setdefault(id(p), (p, []))[1].append(l)
        for p, cons in consumers.values():
            if p.can_write_chunked_residual() and all(c.can_read_chunked_residual() for c in cons):
                p.residual_chunked = True
                for c in cons:
                    c.input_residual_chunked = True

    def part(self, first, n, planes=None):
        """A Network over images [first, first + n) of the live batch: this one's weights, input images and
        logits rows; the activations in between share this one's buffers, and what a producer lays out
        for its consumer (planes) has room of its own, because that layout depends on the batch.
        planes: a dict that parts of the same n which run one after another share theirs through."""
        p = Network.__new__(Network)
        p.spec, p.live_batch = self.spec, n
        p.layers = [l.part(first, n) for l in self.layers]
        p.layers[0].input_gpu = self.layers[0].input_gpu[first:first + n]
        p.layers[-1].output_gpu = self.layers[-1].output_gpu[first:first + n]
        for i, (prod, cons) in enumerate(zip(p.layers, p.layers[1:])):
            if getattr(cons, "input_planes", None) is not None:
                room = None if planes is None else planes.get(i)
                cons.input_planes = ops.new_planes(cons.desc, cons.input_gpu.device) if room is None else room
                if planes is not None:
                    planes[i] = cons.input_planes
                prod.next_layer = (cons.desc, cons.input_planes)
                if cons.pooling_producer is not None:
                    cons.pooling_producer = prod
        p._use_units()
        return p

    def set_input(self, x):
        self.layers[0].set_input(x)

    def set_batch(self, n):
        """Run the following passes on the first n images (n <= the batch the network was built
        for) without rebuilding anything: buffers keep their size, kernels take the live batch.
        The logits of the live images are the first n rows of the output."""
        for l in self.layers:
            l.set_batch(n)
        self._use_units()
        self.live_batch = n

    def kernel_launches(self):
        """Kernels one pass launches."""
        if _Calls(self.layers).chain:
            return 1
        return sum(l.kernel_launches() if hasattr(l, "kernel_launches") else 1 for l in self.layers)

    _pass = None           # of the last call of forward()

    def forward(self):
        """One pass over the layers on the current stream.  A pass that repeats the one before -- the
        same calls on the same buffers -- is recorded as a CUDA graph the third time and replayed from
        then on: the same launches, submitted at once (the MLP's five layers at batch 8 cost the host 21
        us one by one).  Anything that changes a layer's call (a buffer, the live batch, a
        process-wide setting) starts over."""
        p = last = self._pass
        capturing = torch.cuda.is_current_stream_capturing()
        done = last is not None and last.common.hold(self.layers) and not (capturing and last.common.moved())
        if done and p.input != _input_facts(self.layers):
            done = last.common.serves(self.layers[0].input_gpu)
            if done:
                p = self._pass = _Pass(last.common, self.layers, fresh=False)
        if done:
            if not capturing:
                if p.seen == 2:
                    p.graph = p.record()
                p.seen += p.seen < 3
            if p.graph is None or capturing:
                p.run()
            else:
                p.graph.replay()
            done = capturing or not p.common.moved()
        if not done:
            p = self._pass = _Pass(_Calls(self.layers), self.layers)
            p.run()
            if last is not None:                         # (behind the launches: the GPU is busy meanwhile)
                p.common.note(self.layers)
            p.seen = 2 if last is not None and not last.common.noted and last.input == p.input else 1
        return self.layers[-1].get_output_gpu()

    MAX_GRAPHS = 16

    def forward_graph(self):
        """forward() replayed from a CUDA graph: the layer launches (every entry point takes the
        stream and none allocates or synchronises) are captured once per input buffer and live batch, after one
        eager pass that lets the first layer compile its kernel variants, and replayed as one
        submission on the current stream.  Same launches, same results; the host's per-launch
        work and the gaps between the launches go away.  A graph serves while its calls hold (_Calls) and
        keeps the buffers they point into alive; the last MAX_GRAPHS are kept."""
        key = (self.layers[0].input_gpu.data_ptr(), self.live_batch)
        graphs = self.__dict__.setdefault("_graphs", {})
        p = graphs.get(key)
        done = p is not None and p.input == _input_facts(self.layers) and p.common.hold(self.layers)
        if done:
            p.graph.replay()
            done = not p.common.moved()
        if not done:
            p = _Pass(_Calls(self.layers), self.layers)
            p.run()
            p.common.note(self.layers)
            torch.cuda.synchronize()
            p.graph = p.record()
            if p.graph is None:
                raise lib.TcbnnError("the layers' launches could not be recorded as a graph on this stream")
            graphs.pop(key, None)
            while len(graphs) >= self.MAX_GRAPHS:
                graphs.pop(next(iter(graphs)))
            graphs[key] = p
            p.graph.replay()
        return self.layers[-1].get_output_gpu()


class HostFeeder:
    """Feeds a Network from pinned host batches with the host->device copy of batch i+1 running
    on its own stream while batch i is being computed (two device input buffers).  Every batch
    still pays its own copy; only the waiting is overlapped.

    Large batches arrive and are computed in parts: the first compute then waits for a part's copy
    instead of a batch's, and only a part's compute is left once the last copy is done (ResNet-18, three
    batches of 256 byte images, 2090 us of copies: 2742 us by whole batches)."""

    # A part is worth its own pass when copying it takes longer than the layers' latency, about 150 us
    # (16 MiB at 55 GB/s: 305).  At most four: smaller passes fill the GPU less well (128 images of
    # ResNet-18 take 340 us, 256 take 628), and where the compute is the longer side that counts.
    PART_BYTES, MAX_PARTS = 16 << 20, 4

    def __init__(self, net, graph=True):
        """graph: run each forward pass as a CUDA-graph replay (Network.forward_graph)."""
        self.graph = graph
        self.net = net
        self.first = net.layers[0]
        self.bufs = [self.first.input_gpu, torch.empty_like(self.first.input_gpu)]
        self.copy_stream = torch.cuda.Stream()
        self.copied = [torch.cuda.Event(), torch.cuda.Event()]
        self.free = [torch.cuda.Event(), torch.cuda.Event()]
        self.read_stream = torch.cuda.Stream()
        self.computed = torch.cuda.Event()
        self.read_done = torch.cuda.Event()
        self.staged, self.stage_free = [None, None], [torch.cuda.Event(), torch.cuda.Event()]
        self.n = 0
        self.pending = None
        self.part_copied = [[torch.cuda.Event() for _ in range(self.MAX_PARTS)] for _ in range(2)]
        self.cuts = [None, None]                         # how each slot's batch was copied
        # the parts of the network as it is now: (first, n) -> Network.part, and the planes of parts of n
        # images, which run one after another
        self.parts, self.planes, self.parts_of = {}, {}, None

    def _cuts(self):
        """[(first, n)] of the live batch's parts."""
        live = self.net.live_batch or self.net.spec["batch"]
        b = self.bufs[0]
        k = max(1, min(self.MAX_PARTS, live * b[0].numel() * b.element_size() // self.PART_BYTES, live))
        size = (live + k - 1) // k
        return [(f, min(size, live - f)) for f in range(0, live, size)]

    def _enqueue_copy(self, slot, x_host):
        buf = self.bufs[slot]
        x = x_host.reshape(buf.shape)
        cuts = self.cuts[slot] = self._cuts()
        with torch.cuda.stream(self.copy_stream):
            self.copy_stream.wait_event(self.free[slot])
            for i, (first, n) in enumerate(cuts):
                end = buf.shape[0] if i + 1 == len(cuts) else first + n      # (rows behind the live batch too)
                buf[first:end].copy_(x[first:end], non_blocking=True)
                if len(cuts) > 1:
                    self.part_copied[slot][i].record(self.copy_stream)
            self.copied[slot].record(self.copy_stream)

    def _network(self):
        """What a part takes over from the network when it is made."""
        layers = self.net.layers
        return (self.net.live_batch, layers[-1].output_gpu.data_ptr(), [(l, l.state()) for l in layers],
                [bytes(l.desc) for l in layers if hasattr(l, "desc")])

    def _run_parts(self, main, slot, cuts):
        now = self._network()
        if now != self.parts_of:
            self.parts, self.planes, self.parts_of = {}, {}, now
        for i, (first, n) in enumerate(cuts):
            p = self.parts.get((first, n))
            if p is None:
                p = self.parts[(first, n)] = self.net.part(first, n, self.planes.setdefault(n, {}))
            main.wait_event(self.part_copied[slot][i])
            p.layers[0].input_gpu = self.bufs[slot][first:first + n]
            p.forward_graph() if self.graph else p.forward()
        return self.net.layers[-1].get_output_gpu()

    def run(self, batches, on_result=None, result_host=None):
        """batches: iterable of pinned host tensors; on_result(logits_device) is called after
        each forward pass has been queued.  result_host: pinned host tensor that receives every
        batch's logits; that device->host read runs on a third stream, from a copy on the device,
        beside the next batch's compute and input copy."""
        main = torch.cuda.current_stream()
        for ev in self.free:
            ev.record(main)
        self.read_done.record(main)
        it = iter(batches)
        nxt = next(it, None)
        slot = stage = 0
        if nxt is not None:
            self._enqueue_copy(slot, nxt)
        while nxt is not None:
            cur_slot = slot
            nxt = next(it, None)
            if nxt is not None:
                slot ^= 1
                self._enqueue_copy(slot, nxt)
            self.first.input_gpu = self.bufs[cur_slot]
            cuts = self.cuts[cur_slot]
            if len(cuts) > 1 and cuts == self._cuts():
                out = self._run_parts(main, cur_slot, cuts)
            else:                                        # (or the live batch has changed since it was copied)
                main.wait_event(self.copied[cur_slot])
                out = self.net.forward_graph() if self.graph else self.net.forward()
            self.free[cur_slot].record(main)
            if on_result is not None:
                on_result(out)
            if result_host is not None:
                # (two staging buffers: waiting for the read itself, which shares PCIe with the input
                # copies, held the next pass back by 65 us at batch 256)
                main.wait_event(self.stage_free[stage])      # (before its memory can go, too)
                if self.staged[stage] is None or self.staged[stage].shape != out.shape:
                    self.staged[stage] = torch.empty_like(out)
                self.staged[stage].copy_(out)
                self.computed.record(main)
                with torch.cuda.stream(self.read_stream):
                    self.read_stream.wait_event(self.computed)
                    result_host.copy_(self.staged[stage], non_blocking=True)
                    self.stage_free[stage].record(self.read_stream)
                    self.read_done.record(self.read_stream)
                stage ^= 1
        main.wait_event(self.read_done)
