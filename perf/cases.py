"""The work this framework is timed on: whole networks, single layers and the host-fed pipeline, called
through the public entry points (models.Network, models.HostFeeder, ops.*).

A case is a dict of plain values; "kind" picks what it runs:

  net   one forward pass of a network topology of models.py, inputs resident on the GPU
  feed  a run of HostFeeder over batches in pinned host memory (bytes in, logits out)
  gemm  one bit GEMM: int32 sums, threshold bits (hidden layer) or scale + bias (output layer)
  conv  one binary convolution layer called by itself, with its residual and pooling options

Sizes are those of the reference drivers' networks, of BASELINE's five configurations, and of the
tests and the microbenchmark; all data is synthetic.
"""
import math

import torch

from tcbnn_b200 import models, ops


# ---- the cases -----------------------------------------------------------------------------------

def _net(topology, batch, live=None, u8=False, bound=False, graph=False):
    """live: images of the pass (set_batch) on a network built for `batch`.  u8: images arrive as
    bytes with their value table.  bound: the caller states max |pixel|, so that residuals can be
    int16.  graph: forward_graph() instead of forward()."""
    return dict(kind="net", topology=topology, batch=batch, live=live or batch, u8=u8, bound=bound, graph=graph)


def _conv(B, hw, C, O, filt=3, stride=1, pool=1, residual="none", save="none"):
    """residual / save: element type of the residual tensor injected / saved ("none", "int16", "int32")."""
    return dict(kind="conv", B=B, hw=hw, C=C, O=O, filter=filt, stride=stride, pool=pool, residual=residual, save=save)


def listed():
    return [
        # an interactive request to the MNIST MLP: five short layers, nothing but latency
        dict(_net("mlp", 8), name="mlp_b8"),
        # the MLP scoring a large batch
        dict(_net("mlp", 8192), name="mlp_b8192"),
        # the CIFAR VGG at its batch: pooled layers, three FC layers
        dict(_net("vgg_cifar", 1024), name="vgg_cifar_b1024"),
        # the last, ragged batch of an evaluation loop on the CIFAR ResNet; the caller states no bound
        # of its pixels, so the shortcut sums are int32
        dict(_net("resnet_cifar", 256, live=201), name="resnet_cifar_live201"),
        # one camera image through ResNet-18: latency, every layer far too small for the GPU
        dict(_net("resnet18", 1, u8=True, bound=True, graph=True), name="resnet18_b1"),
        # the headline: ResNet-18 at batch 1024
        dict(_net("resnet18", 1024, bound=True, graph=True), name="resnet18_b1024"),
        # VGG-16 at 224 x 224: wide pooled layers on large images, 4096-wide FC layers
        dict(_net("vgg16_imagenet", 32), name="vgg16_imagenet_b32"),
        # ResNet-18 fed from pinned host memory: three batches of bytes in, logits out
        dict(kind="feed", batch=256, batches=3, name="resnet18_feed_b256"),
        # the standalone bit GEMM
        dict(kind="gemm", M=1024, N=1024, K=4096, mode="int32", name="gemm_1024x1024x4096"),
        # the first FC layer of AlexNet on a ragged batch
        dict(kind="gemm", M=777, N=4096, K=9216, mode="bits", name="fc_777x4096x9216"),
        # the standalone convolution, its integer result saved
        dict(_conv(256, 56, 128, 128, save="int32"), name="conv_56x56x128_b256"),
        # the 5 x 5 pooled layer of AlexNet
        dict(_conv(100, 28, 64, 192, filt=5, pool=2), name="conv_5x5_pooled_b100"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        p = rng.random()
        if p < 0.4:
            top, most = rng.choice([("mlp", 8192), ("mlp", 8192), ("vgg_cifar", 1024), ("resnet_cifar", 512),
                                    ("resnet18", 1024), ("vgg16_imagenet", 32)])
            batch = _log(rng, 1, most)
            image, resnet = top != "mlp", top.startswith("resnet")
            return _net(top, batch, live=rng.randint(max(1, batch // 2), batch) if rng.random() < 0.3 else batch,
                        u8=image and rng.random() < 0.4, bound=resnet and rng.random() < 0.6, graph=rng.random() < 0.4)
        if p < 0.45:
            return dict(kind="feed", batch=_log(rng, 16, 256), batches=rng.randint(2, 4))
        if p < 0.72:
            mode = rng.choice(["int32", "bits", "affine"])
            N = _log(rng, 10, 1000) if mode == "affine" else _log(rng, 64, 8192)
            return dict(kind="gemm", M=_log(rng, 1, 8192), N=N, K=_log(rng, 64, 16384), mode=mode)
        C, O = (rng.choice([64, 64, 128, 128, 192, 256, 256, 384, 512, 512]) for _ in range(2))
        filt, stride = rng.choice([(3, 1)] * 5 + [(3, 2)] * 2 + [(5, 1), (1, 1)])
        pool = 2 if stride == 1 and rng.random() < 0.25 else 1
        hw = _log(rng, 7, 112)
        if (stride == 2 or pool == 2) and hw % 2:
            hw += 1
        res, save = ("none", "none") if pool == 2 else rng.choice(
            [("none", "none"), ("none", "none"), ("none", "int16"), ("int16", "int16"), ("int32", "int32"), ("none", "int32")])
        c = _conv(_log(rng, 1, 512), hw, C, O, filt, stride, pool, res, save)
        w = work(c)
        if w["flops"] <= 2.5e12 and w["bytes"] <= 2e9:
            return c


# ---- inputs and what a program keeps ---------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _words(shape, g):
    return torch.randint(-2 ** 31, 2 ** 31, shape, dtype=torch.int64, device="cuda", generator=g).to(torch.int32)


def _spec(case):
    return getattr(models, case["topology"] + "_spec")(case["batch"])


def _weights(spec, g):
    """models.synthetic_weights drawn on the GPU: +-1 weights, thresholds N(0, sqrt(fan_in))."""
    arrays = []

    def pm1(*shape):
        arrays.append(torch.randint(0, 2, shape, dtype=torch.int8, device="cuda", generator=g).float().mul_(2).sub_(1))

    def normal(n, scale, shift=0.0):
        arrays.append(torch.randn(n, device="cuda", generator=g) * scale + shift)

    for l in models.layer_shapes(spec):
        if l["type"] in ("inconv", "conv"):
            pm1(l["R"] * l["S"], l["C"], l["O"])
            normal(l["O"], math.sqrt(l["R"] * l["S"] * l["C"]))
        elif l["type"] in ("fc", "out"):
            pm1(l["K"], l["N"])
            if l["type"] == "fc":
                normal(l["N"], math.sqrt(l["K"]))
            else:
                normal(l["N"], 0.1, 1.0)
                normal(l["N"], 1.0)
    return [a.cpu().numpy() for a in arrays]


_MEAN, _STD = (0.485, 0.456, 0.406), (0.229, 0.224, 0.225)


def _images(batch, first, g):
    return torch.randint(0, 256, (batch, 3, first["H"], first["W"]), dtype=torch.uint8, device="cuda", generator=g)


def _table():
    """fp32 value of every byte per channel: the readers' normalisation."""
    v = torch.arange(256, dtype=torch.float32).reshape(1, 256) / 255.0
    return ((v - torch.tensor(_MEAN).reshape(3, 1)) / torch.tensor(_STD).reshape(3, 1)).numpy()


def _build(spec, g, u8, bound):
    first = spec["layers"][0]
    weights = _weights(spec, g)
    lut = None
    if first["type"] == "in":
        x = torch.rand((spec["batch"], first["K"]), device="cuda", generator=g) - 0.5
    else:
        x = _images(spec["batch"], first, g)
        if u8:
            lut = _table()
        else:
            mean, std = (torch.tensor(t, device="cuda").reshape(1, 3, 1, 1) for t in (_MEAN, _STD))
            x = (x.float() / 255.0 - mean) / std
    return models.Network(spec, weights, x, input_abs_bound=models.SYNTHETIC_IMAGE_ABS_BOUND if bound else None, input_lut=lut)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "net":
        net = _build(_spec(case), g, case["u8"], case["bound"])
        if case["live"] != case["batch"]:
            net.set_batch(case["live"])
        return dict(case=case, net=net)
    if kind == "feed":
        spec = models.resnet18_spec(case["batch"])
        net = _build(spec, g, True, True)
        batches = []
        for _ in range(case["batches"]):
            h = torch.empty((case["batch"], 3, 224, 224), dtype=torch.uint8, pin_memory=True)
            h.copy_(_images(case["batch"], spec["layers"][0], g))
            batches.append(h)
        logits = torch.empty((case["batch"], 1000), dtype=torch.float32, pin_memory=True)
        return dict(case=case, feeder=models.HostFeeder(net), batches=batches, logits=logits)
    if kind == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        ld = ops.step128_words(K)
        keep = torch.full((ld,), -1, dtype=torch.int32, device="cuda")      # bits past K are 0
        keep[(K + 31) // 32:] = 0
        if K % 32:
            keep[K // 32] = -(1 << (32 - K % 32))
        return dict(case=case, a=_words((M, ld), g) & keep, w=_words((N, ld), g) & keep,
                    p0=torch.randn(N, device="cuda", generator=g) * math.sqrt(K), p1=torch.randn(N, device="cuda", generator=g),
                    workspace=ops.gemm_workspace(M, N, K, torch.device("cuda", torch.cuda.current_device())))
    B, hw, C, O, R = case["B"], case["hw"], case["C"], case["O"], case["filter"]
    d = ops.conv_desc(B, hw, hw, C, O, R, R, case["stride"], case["stride"], pool=case["pool"])
    residual = None
    if case["residual"] != "none":
        residual = torch.randint(-1500, 1501, (B, d.OH, d.OW, O), device="cuda", generator=g,
                                 dtype=getattr(torch, case["residual"]))
    return dict(case=case, d=d, x=_words((B, hw, hw, C // 32), g), filt=ops.conv_prepare(d, _words((O, R * R, C // 32), g)),
                thr=torch.randn(O, device="cuda", generator=g) * math.sqrt(R * R * C), residual=residual)


# ---- one pass ------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "net":
        net = state["net"]
        return (net.forward_graph() if case["graph"] else net.forward())[:case["live"]]
    if kind == "feed":
        got = []
        state["feeder"].run(state["batches"], on_result=lambda logits: got.append(logits.clone()), result_host=state["logits"])
        return got + [state["logits"]]
    if kind == "gemm":
        a, w, K, ws = state["a"], state["w"], case["K"], state["workspace"]
        if case["mode"] == "int32":
            return ops.bgemm(a, w, K, workspace=ws)
        if case["mode"] == "bits":
            return ops.fc_layer(a, w, state["p0"], K, workspace=ws)
        return ops.out_layer(a, w, state["p0"], state["p1"], K, workspace=ws)
    save, residual = case["save"], state["residual"]
    out, saved, _ = ops.conv_layer(state["d"], state["x"], state["filt"], state["thr"], res_in=residual,
                                   residual_channels=case["O"] if residual is not None else 0,
                                   save_residual=save != "none", residual_dtype=torch.int16 if save == "int16" else torch.int32)
    return out if saved is None else (out, saved)


# ---- what a pass cannot do without ------------------------------------------------------------------

def _elem(name):
    return {"none": 0, "int16": 2, "int32": 4}[name]


def _net_work(spec, live, pixel_bytes):
    """Input, packed weights and logits once; two operations per multiply-accumulate (per addition
    of a pixel value in the first layer)."""
    nbytes = flops = 0
    for l in models.layer_shapes(spec):
        if l["type"] == "in":
            nbytes += live * l["K"] * 4
        elif l["type"] in ("inconv", "conv"):
            taps = l["R"] * l["S"] * l["C"]
            flops += 2 * live * l["OH"] * l["OW"] * l["pool"] ** 2 * l["O"] * taps
            nbytes += l["O"] * taps // 8 + 4 * l["O"] + (live * 3 * l["H"] * l["W"] * pixel_bytes if l["type"] == "inconv" else 0)
        else:
            flops += 2 * live * l["K"] * l["N"]
            nbytes += l["K"] * l["N"] // 8 + 4 * l["N"]
            last = l["N"]
    return dict(bytes=nbytes + 4 * live * last, flops=flops)


def work(case):
    kind = case["kind"]
    if kind == "net":
        return _net_work(_spec(case), case["live"], 1 if case["u8"] else 4)
    if kind == "feed":
        n = case["batch"] * case["batches"]
        return _net_work(models.resnet18_spec(case["batch"]), n, 1)
    if kind == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        out = M * ((N + 31) // 32) * 4 if case["mode"] == "bits" else M * N * 4
        return dict(bytes=(M + N) * ((K + 31) // 32) * 4 + out + 4 * N, flops=2 * M * N * K)
    B, hw, C, O, taps = case["B"], case["hw"], case["C"], case["O"], case["filter"] ** 2
    grid = B * ((hw + case["stride"] - 1) // case["stride"]) ** 2            # before pooling
    return dict(bytes=B * hw * hw * C // 8 + O * taps * C // 8 + 4 * O + grid // case["pool"] ** 2 * O // 8 +
                grid * O * (_elem(case["residual"]) + _elem(case["save"])),
                flops=2 * grid * O * taps * C)


def tolerance(case):
    """Packed bits and integers are exact; logits are one fp32 multiply-add on exact integers."""
    if case["kind"] in ("net", "feed") or case.get("mode") == "affine":
        return {"rel": 1e-5, "max": 1e-4}
    return "exact"
