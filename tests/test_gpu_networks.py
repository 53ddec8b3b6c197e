"""GPU parity of whole networks, layer by layer, against the CPU oracle."""
import gc
import weakref

import numpy as np
import pytest
import torch

import networks as onet
import util
from tcbnn_b200 import lib, models, ops

pytestmark = pytest.mark.gpu


def _compare(spec, seed, cuda, input_abs_bound=None):
    w = models.synthetic_weights(spec, seed)
    x = models.synthetic_input(spec, seed + 1)
    acts, ress = onet.run(spec, w, x)
    net = models.Network(spec, w, x, input_abs_bound=input_abs_bound)
    logits = net.forward()
    torch.cuda.synchronize()
    for i, (layer, a, r) in enumerate(zip(net.layers, acts, ress)):
        got = layer.get_output_gpu().cpu().numpy()
        if got.dtype == np.int32:
            got = got.view(np.uint32)
            assert np.array_equal(got.reshape(a.shape), a), "layer %d %s bits" % (i, layer.name)
        if r is not None:
            if input_abs_bound is not None:
                assert layer.get_output_residual_gpu().dtype == torch.int16
            gr = layer.download_output_residual()          # int32 NHWC whatever the device layout
            assert np.array_equal(gr, r), "layer %d %s residual" % (i, layer.name)
    ref = acts[-1]
    got = logits.cpu().numpy()
    np.testing.assert_allclose(got, ref, rtol=1e-5, atol=1e-5)
    # a second pass over the same objects gives the same logits (layers store, never OR)
    again = net.forward().cpu().numpy()
    assert np.array_equal(again, got)


def test_mlp(cuda):
    _compare(models.mlp_spec(256), 5, cuda)


@pytest.mark.parametrize("batch, widths", [(1401, (784, 1031, 999, 1100)), (1400, (845, 1024, 928, 1500))])
def test_fc_layers_hand_their_operands_over_expanded(cuda, batch, widths):
    # ragged rows and columns (words and k-blocks half used), either packing kernel of the input layer
    spec = models.mlp_spec(batch, widths[0])
    for l, n in zip(spec["layers"][1:-1], widths[1:]):
        l["N"] = n
    _compare(spec, 17, cuda)
    w, x = models.synthetic_weights(spec, 17), models.synthetic_input(spec, 18)
    net = models.Network(spec, w, x)
    assert all(l.input_units is not None for l in net.layers[1:-1])
    want = net.forward().clone()
    net.set_batch(batch - 200)                       # other rows of the last tile, or another kernel
    assert torch.equal(net.forward()[:batch - 200], want[:batch - 200])
    net.set_batch(40)
    assert torch.equal(net.forward()[:40], want[:40])
    net.set_batch(batch)
    fc = net.layers[2]
    fc.weight_gpu.copy_(torch.zeros_like(fc.weight_gpu))       # a weight written to in place counts
    changed = net.forward().clone()
    plain = models.Network(spec, w, x, handover=False)
    plain.layers[2].weight_gpu.zero_()
    assert torch.equal(changed, plain.forward()) and not torch.equal(changed, want)


def _write(how, t, new):
    """`new` into tensor `t`, by a torch operation, past torch's version counter, or by this library."""
    if how == "copy_":
        t.copy_(new)
    elif how == "data":
        t.data.copy_(new)
    else:
        ops.fc_layer(new, torch.zeros((t.shape[1] * 32, 4), dtype=torch.int32, device=t.device),
                     torch.zeros(t.shape[1] * 32, device=t.device), 128, out=t)


def _fc_chain(batch=1400):
    """Two FC layers on the tcgen05 GEMM between an input layer and the output layer, and other weights."""
    spec = models.mlp_spec(batch)
    w = models.synthetic_weights(spec, 31)
    return spec, w, models.synthetic_input(spec, 32), models.synthetic_weights(spec, 33)


@pytest.mark.parametrize("path", ["forward", "forward_graph", "feeder", "feeder_parts"])
@pytest.mark.parametrize("how", ["copy_", "data", "library", "inference"])
def test_fc_weights_written_between_passes_count(cuda, how, path):
    """Whatever writes a packed weight between two passes is followed by the next one: on the call paths of
    a network, its replayed passes and the feeder's, whole batches and parts."""
    spec, w, x, other = _fc_chain(2800 if path == "feeder_parts" else 1400)      # (parts of 1400)
    with torch.inference_mode(how == "inference"):
        net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
        assert all(l.weight_units is not None and l.reads_units for l in net.layers[2:4])
        host = torch.from_numpy(x).pin_memory()
        feeder = models.HostFeeder(net)
        if path == "feeder_parts":
            feeder.PART_BYTES = x.nbytes // 2
        def run():
            if path.startswith("feeder"):
                got = []
                feeder.run([host], lambda out: got.append(out.clone()))
                return got[0]
            return getattr(net, path)().clone()
        want = plain.forward().clone()
        for _ in range(4):                           # (forward() replays a graph by then)
            assert torch.equal(run(), want)
        g = util.rng(34)
        for i in (2, 3):
            t = net.layers[i].weight_gpu
            if how == "library":                     # bits of an FC layer, N = K of the weight's rows
                src = torch.from_numpy(util.rand_words(g, (t.shape[0], 4)).view(np.int32)).to(cuda)
                _write(how, t, src)
            else:
                new = ops.pack_fc_weight(torch.from_numpy(other[2 * i - 2].reshape(1024, 1024)).to(cuda))
                _write("copy_" if how == "inference" else how, t, new)
            plain.layers[i].weight_gpu.copy_(t)
        changed = plain.forward().clone()
        assert not torch.equal(changed, want)
        for _ in range(3):
            assert torch.equal(run(), changed)


@pytest.mark.parametrize("how", ["copy_", "data", "library"])
def test_layer_called_by_itself_reads_its_input_rows(cuda, how):
    """A layer object's own forward() computes from the packed rows in input_gpu, whoever wrote them last."""
    spec, w, x, _ = _fc_chain()
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    net.forward()
    before = net.layers[2].get_output_gpu().clone()
    rows = net.layers[1].get_output_gpu()
    g = util.rng(35)
    words = 4 if how == "library" else rows.shape[1]
    _write(how, rows, torch.from_numpy(util.rand_words(g, (rows.shape[0], words)).view(np.int32)).to(cuda))
    plain.layers[1].get_output_gpu().copy_(rows)
    net.layers[2].forward()
    plain.layers[2].forward()
    assert torch.equal(net.layers[2].get_output_gpu(), plain.layers[2].get_output_gpu())
    assert not torch.equal(net.layers[2].get_output_gpu(), before)


@pytest.mark.parametrize("which", ["mlp", "resnet18"])
def test_tensor_given_another_storage_in_place_counts(cuda, which):
    """layer.tensor.data = other moves a tensor under its layer: the next pass uses the new storage, replayed
    passes and single calls alike.  (The old storage is kept alive throughout.)"""
    spec = models.mlp_spec(8) if which == "mlp" else models.resnet18_spec(2, image=64, classes=100)
    w, x = models.synthetic_weights(spec, 40), models.synthetic_input(spec, 41)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    for _ in range(4):
        want = net.forward().clone()
    old = []
    for i in ((1, 3) if which == "mlp" else (4, len(spec["layers"]) - 2)):
        for n in (net, plain):
            t = n.layers[i].bn_gpu
            old.append(t.detach())
            t.data = t + 9.0
    changed = plain.forward().clone()
    assert not torch.equal(changed, want)
    for _ in range(4):
        assert torch.equal(net.forward(), changed)
    i = 3 if which == "mlp" else 4
    for n in (net, plain):
        t = n.layers[i].bn_gpu
        old.append(t.detach())
        t.data = t - 20.0
        n.layers[i].forward()
    assert torch.equal(net.layers[i].get_output_gpu(), plain.layers[i].get_output_gpu())
    fc = next(l for l in net.layers if type(l).__name__ == "Fc128LayerParam")
    assert fc.weight_gpu.shape[0] > 4
    fc.weight_gpu.t_()
    with pytest.raises(lib.TcbnnError):              # refused as it always was: rows are no longer contiguous
        net.forward()


@pytest.mark.parametrize("which", ["mlp", "vgg_cifar"])
def test_network_gives_its_memory_back_when_dropped(cuda, which):
    """Layers, buffers and recorded passes form no reference cycle: what a network holds is free as soon as the
    last reference to it goes, not when the garbage collector gets to it."""
    spec = models.mlp_spec(1100) if which == "mlp" else models.vgg_cifar_spec(4)
    w, x = models.synthetic_weights(spec, 70), models.synthetic_input(spec, 71)
    gc.collect()
    gc.disable()
    try:
        net = models.Network(spec, w, x)
        feeder = models.HostFeeder(net)
        feeder.PART_BYTES = x.nbytes // 2
        for _ in range(4):
            net.forward()
        net.forward_graph()
        feeder.run([torch.from_numpy(np.ascontiguousarray(x)).pin_memory()])
        torch.cuda.synchronize()
        gone = [weakref.ref(l) for l in net.layers] + [weakref.ref(p) for p in feeder.parts.values()]
        del net, feeder
        assert all(r() is None for r in gone)
    finally:
        gc.enable()


def test_live_batches_that_come_back_replay_their_graphs(cuda):
    spec = models.vgg_cifar_spec(6)
    net = models.Network(spec, models.synthetic_weights(spec, 72), models.synthetic_input(spec, 73))
    want = net.forward().clone()
    kept = {}
    for live in (6, 5, 6, 5, 6):
        net.set_batch(live)
        assert torch.equal(net.forward_graph()[:live], want[:live])
        p = net._graphs[(net.layers[0].input_gpu.data_ptr(), live)]
        assert kept.setdefault(live, p) is p


@pytest.mark.parametrize("which", ["mlp", "resnet18", "vgg_cifar"])
def test_forward_replays_follow_inputs_and_every_change(cuda, which):
    """forward() replays a recorded graph from its third call on: on new images each time, and after each of
    the things that end a replay, its logits are those of the layers called one by one."""
    spec = {"mlp": models.mlp_spec(1100), "resnet18": models.resnet18_spec(3, image=64, classes=100),
            "vgg_cifar": models.vgg_cifar_spec(5)}[which]
    w, bound = models.synthetic_weights(spec, 60), models.SYNTHETIC_IMAGE_ABS_BOUND if which == "resnet18" else None
    net = models.Network(spec, w, models.synthetic_input(spec, 61), input_abs_bound=bound)
    xs = [torch.from_numpy(models.synthetic_input(spec, 62 + i)).to(cuda) for i in range(5)]
    B = spec["batch"]

    def check(live=B):
        seen = set()
        for x in xs:
            net.set_input(x[:live])
            got = net.forward()[:live].clone()
            replays = net._pass.graph is not None
            for l in net.layers:
                l.forward()
            want = net.layers[-1].get_output_gpu()[:live]
            assert torch.equal(got, want)
            seen.add(bytes(want.cpu().numpy()))
        assert replays and len(seen) == len(xs)             # the last of them at least was a replay

    try:
        check()
        for change in ("weight", "thresholds", "settings", "plan", "live", "input", "scratch"):
            if change == "weight":
                net.layers[-1].weight_gpu.copy_(net.layers[-1].weight_gpu.flip(0))
            elif change == "thresholds":
                net.layers[2].bn_gpu = net.layers[2].bn_gpu - 3.0
            elif change == "settings":
                ops.set_conv_path(6)
                check()
                ops.set_conv_path(0)
            elif change == "plan":
                ops.set_gemm_plan(1, 1)
                check()
                ops.set_gemm_plan(-1, -1)
            elif change == "live":
                net.set_batch(B - 1)
                check(B - 1)
                net.set_batch(B)
            elif change == "input":
                net.layers[0].input_gpu = torch.empty_like(net.layers[0].input_gpu)
            elif ops.shared_scratch(net.layers[0].output_gpu.device) is not None:
                ops.conv_workspace(ops.conv_desc(96, 32, 32, 128, 128, 3, 3, 1, 1, pool=2), net.layers[0].output_gpu.device)
            check()
    finally:
        ops.set_conv_path(0)
        ops.set_gemm_plan(-1, -1)


def test_graph_is_recorded_again_when_its_pass_has_changed(cuda):
    """forward_graph() after a layer's tensor was replaced, after a process-wide setting changed and for live
    batches that come back: the results of a network without graphs.  The graphs kept are bounded."""
    spec = models.mlp_spec(40)
    w, x = models.synthetic_weights(spec, 42), models.synthetic_input(spec, 43)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    want = net.forward_graph().clone()
    kept = [t for n in (net, plain) for t in (n.layers[2].bn_gpu, n.layers[3].weight_gpu)]     # (whoever reads these is caught)
    for n in (net, plain):
        n.layers[2].bn_gpu = n.layers[2].bn_gpu + 9.0
        n.layers[3].weight_gpu = n.layers[3].weight_gpu.flip(0).contiguous()
    changed = plain.forward().clone()
    assert torch.equal(net.forward_graph(), changed) and not torch.equal(changed, want) and len(kept) == 4
    net.MAX_GRAPHS = 3
    for live in (40, 33, 7, 12, 40, 33):
        net.set_batch(live)
        assert torch.equal(net.forward_graph()[:live], changed[:live])
        assert len(net._graphs) <= 3
    held = net._graphs[next(reversed(net._graphs))]
    ops.set_conv_path(6)
    try:
        assert torch.equal(net.forward_graph()[:33], changed[:33])
        assert net._graphs[next(reversed(net._graphs))] is not held
    finally:
        ops.set_conv_path(0)


def test_passes_back_to_back_on_shared_scratch(cuda):
    """Passes queued one behind the other on changing images, every layer expanding its input and pooling its
    output through the one scratch: each pass's logits are those of a pass with nothing around it."""
    spec = models.vgg_cifar_spec(37)
    net = models.Network(spec, models.synthetic_weights(spec, 52), models.synthetic_input(spec, 53), handover=False)
    xs = [torch.from_numpy(models.synthetic_input(spec, 54 + i)).to(cuda) for i in range(3)]
    alone = []
    for x in xs:
        net.set_input(x)
        alone.append(net.forward().clone())
        torch.cuda.synchronize()
    assert not torch.equal(alone[0], alone[1])
    got = []
    for i in range(60):
        net.set_input(xs[i % 3])
        got.append((net.forward_graph() if i >= 30 else net.forward()).clone())
    assert all(torch.equal(g, alone[i % 3]) for i, g in enumerate(got))


def test_graph_keeps_off_scratch_that_was_replaced(cuda):
    """The scratch shared by layers without planes grows for a larger layer: a graph recorded before that must
    not write to the old one's memory, which by then belongs to somebody else."""
    spec = models.vgg_cifar_spec(2)
    w, x = models.synthetic_weights(spec, 44), models.synthetic_input(spec, 45)
    torch.cuda.synchronize()
    ops._scratch.clear()
    torch.cuda.empty_cache()
    net = models.Network(spec, w, x, handover=False)
    net.set_batch(2)
    want = net.forward_graph().clone()
    size = ops.shared_scratch(cuda if cuda.index is not None else torch.device("cuda", 0)).numel()
    d = ops.conv_desc(64, 32, 32, 128, 128, 3, 3, 1, 1)
    assert ops.conv_workspace(d, torch.device("cuda", 0)).numel() > size
    net.set_batch(1)                                # drops the layers' own hold on the old scratch
    net.set_batch(2)
    others = [torch.full((size,), 7, dtype=torch.uint8, device=cuda) for _ in range(3)]
    for _ in range(2):
        assert torch.equal(net.forward_graph(), want)
    assert all(bool((t == 7).all()) for t in others)


@pytest.mark.parametrize("replaced", [False, True])
def test_conv_behind_pooling_layer_follows_its_input_rows(cuda, replaced):
    """A convolution behind a pooling layer, called by itself after its input rows were written to; and in a
    pass after the producer was given another output tensor (the consumer keeps reading its own)."""
    spec = models.vgg_cifar_spec(3)
    w, x = models.synthetic_weights(spec, 36), models.synthetic_input(spec, 37)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    i = 1 + next(k for k, l in enumerate(net.layers) if type(l).__name__ == "Conv128LayerParam" and l.desc.pool == 2)
    assert net.layers[i].input_planes is not None
    net.forward()
    before = net.layers[i].get_output_gpu().clone()
    rows = net.layers[i - 1].get_output_gpu()
    new = torch.from_numpy(util.rand_words(util.rng(38), tuple(rows.shape)).view(np.int32)).to(cuda)
    for n in (net, plain):
        if replaced:
            n.layers[i - 1].output_gpu = torch.zeros_like(rows)
        n.layers[i].input_gpu.copy_(new.reshape(n.layers[i].input_gpu.shape))
        n.forward() if replaced else n.layers[i].forward()
    assert torch.equal(net.layers[i].get_output_gpu(), plain.layers[i].get_output_gpu())
    assert not torch.equal(net.layers[i].get_output_gpu(), before)


def test_vgg_cifar(cuda):
    _compare(models.vgg_cifar_spec(8), 10, cuda)


def test_alexnet_small_image(cuda):
    # alexnet.cu topology (11x11/4 + pool, 5x5 + pool, 192 / 384 channels) on 96x96 images
    _compare(models.alexnet_spec(4, image=96, hidden=256, classes=100), 40, cuda)


def test_vgg16_imagenet_small_image(cuda):
    # imagenet_vgg.cu topology (13 conv layers, five of them pooled) on 32x32 images
    _compare(models.vgg16_imagenet_spec(3, image=32, hidden=256, classes=100), 50, cuda)


def test_resnet18_small_image(cuda):
    # same topology, 64x64 input -> 16x16 ... 2x2 feature maps
    _compare(models.resnet18_spec(8, image=64, classes=100), 20, cuda)


def test_resnet18_224(cuda):
    _compare(models.resnet18_spec(2), 30, cuda)


def test_resnet18_224_int16_residuals(cuda):
    # same network with the stated input bound: residual chain stored as int16, values identical
    _compare(models.resnet18_spec(3), 31, cuda, input_abs_bound=models.SYNTHETIC_IMAGE_ABS_BOUND)


def test_resnet18_chunked_residual_layout_is_wired_where_it_pays(cuda):
    """With int16 residuals every residual tensor of the network (first layer -> ... -> L4B1C2; the
    last block saves none) is kept in the chunk-major layout: all its producers and consumers run
    the loader-fed kernel, whose tile-per-group epilogue takes that layout only; pooled ones are
    then read in place, so no layer launches a pooling pass."""
    spec = models.resnet18_spec(2)
    net = models.Network(spec, models.synthetic_weights(spec, 32), models.synthetic_input(spec, 33),
                         input_abs_bound=models.SYNTHETIC_IMAGE_ABS_BOUND)
    by = {l.name: l for l in net.layers}
    assert by["Conv1"].residual_chunked
    for stage in "1234":
        for block in "12":
            l = by["L%sB%sC2" % (stage, block)]
            assert l.input_residual_chunked, l.name
            if l.output_residual_gpu is not None:
                assert l.residual_chunked, l.name
            assert l.kernel_launches() == 1, l.name


def test_resnet18_both_conv_kernels(cuda):
    from tcbnn_b200 import ops
    try:
        ops.set_conv_path(1)                 # warp-level b1 MMA everywhere
        _compare(models.resnet18_spec(2, image=64, classes=100), 21, cuda)
    finally:
        ops.set_conv_path(0)


def test_resnet18_uint8_images_give_identical_results(cuda):
    """Byte images + per-channel value table through tcbnn_inconv_layer_u8: every tensor equal
    to the fp32-image run of the same network."""
    spec = models.resnet18_spec(3)
    w = models.synthetic_weights(spec, 50)
    x = models.synthetic_input(spec, 51)
    u8, lut = models.synthetic_input_u8(spec, 51)
    assert np.array_equal(lut[np.arange(3)[None, :, None, None], u8], x)       # same pixels
    ref = models.Network(spec, w, x)
    got = models.Network(spec, w, torch.from_numpy(u8), input_lut=lut)
    a, b = ref.forward().cpu().numpy(), got.forward().cpu().numpy()
    for la, lb in zip(ref.layers, got.layers):
        assert torch.equal(la.get_output_gpu(), lb.get_output_gpu()), la.name
    assert np.array_equal(a, b)
    acts, _ = onet.run(spec, w, x)
    np.testing.assert_allclose(b, acts[-1], rtol=1e-5, atol=1e-5)


def test_forward_graph_replay_equals_eager_forward(cuda):
    """Network.forward_graph: the same launches captured into a CUDA graph; replays follow the
    contents of the input buffer and give the eager results bit for bit."""
    spec = models.resnet18_spec(4, image=64, classes=100)
    w = models.synthetic_weights(spec, 60)
    x0 = models.synthetic_input(spec, 61)
    x1 = models.synthetic_input(spec, 62)
    net = models.Network(spec, w, x0, input_abs_bound=models.SYNTHETIC_IMAGE_ABS_BOUND)
    eager0 = net.forward().clone()
    g0 = net.forward_graph().clone()            # captures
    assert torch.equal(g0, eager0)
    net.layers[0].input_gpu.copy_(torch.from_numpy(x1).to(cuda).reshape(net.layers[0].input_gpu.shape))
    g1 = net.forward_graph().clone()            # replays on the new images
    eager1 = net.forward().clone()
    assert torch.equal(g1, eager1) and not torch.equal(g1, g0)
    acts, _ = onet.run(spec, w, x1)
    np.testing.assert_allclose(g1.cpu().numpy(), acts[-1], rtol=1e-5, atol=1e-5)


def test_host_feeder_overlapped_copies_give_each_batch_its_own_logits(cuda):
    """models.HostFeeder: pinned host batches in, input copy of batch i+1 and logits read of
    batch i beside the compute of the batch between them; every batch's logits equal those of
    a plain forward pass on that batch, with and without graph replay."""
    spec = models.resnet18_spec(4, image=64, classes=100)
    w = models.synthetic_weights(spec, 70)
    xs = [models.synthetic_input(spec, 71 + i) for i in range(4)]
    expect = []
    for x in xs:
        expect.append(models.Network(spec, w, x, input_abs_bound=models.SYNTHETIC_IMAGE_ABS_BOUND).forward().cpu().numpy())
    for graph in (False, True):
        net = models.Network(spec, w, xs[0], input_abs_bound=models.SYNTHETIC_IMAGE_ABS_BOUND)
        feeder = models.HostFeeder(net, graph=graph)
        host = [torch.from_numpy(np.ascontiguousarray(x)).pin_memory() for x in xs]
        last = torch.empty((4, 100), dtype=torch.float32).pin_memory()
        got = []
        feeder.run(host, lambda out: got.append(out.clone()), last)
        torch.cuda.synchronize()
        assert len(got) == len(xs)
        for g, e in zip(got, expect):
            assert np.array_equal(g.cpu().numpy(), e)
        assert np.array_equal(last.numpy(), expect[-1])


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("which,parts", [("resnet18", 2), ("resnet18", 5), ("vgg_cifar", 3), ("mlp", 2)])
def test_host_feeder_computes_large_batches_in_parts(cuda, which, parts, graph):
    """Large batches are computed part by part (two even parts, a shorter last one, one image each)
    behind their copies: every batch's logits equal the whole-batch pass's, on two runs of one feeder."""
    spec = {"resnet18": models.resnet18_spec(5, image=64, classes=100), "vgg_cifar": models.vgg_cifar_spec(7),
            "mlp": models.mlp_spec(6)}[which]
    bound = models.SYNTHETIC_IMAGE_ABS_BOUND if which == "resnet18" else None
    w = models.synthetic_weights(spec, 75)
    xs = [np.ascontiguousarray(models.synthetic_input(spec, 76 + i)) for i in range(2)]
    expect = [models.Network(spec, w, x, input_abs_bound=bound).forward().cpu().numpy() for x in xs]
    feeder = models.HostFeeder(models.Network(spec, w, xs[0], input_abs_bound=bound), graph=graph)
    feeder.PART_BYTES = xs[0].nbytes // parts
    feeder.MAX_PARTS = 5
    feeder.part_copied = [[torch.cuda.Event() for _ in range(5)] for _ in range(2)]
    assert len(feeder._cuts()) == parts
    for _ in range(2):
        got = []
        last = torch.empty(expect[0].shape, dtype=torch.float32).pin_memory()
        feeder.run([torch.from_numpy(x).pin_memory() for x in xs], lambda out: got.append(out.clone()), last)
        torch.cuda.synchronize()
        assert all(np.array_equal(g.cpu().numpy(), e) for g, e in zip(got, expect))
        assert np.array_equal(last.numpy(), expect[-1])


@pytest.mark.parametrize("graph", [False, True])
def test_host_feeder_parts_follow_the_network(cuda, graph):
    """Between two runs a layer is given other thresholds, the logits tensor another storage, and from a
    batch's callback, with the next batch copied in parts already, the live batch changes.  Parts of
    the same size share their planes, and none is kept of a network that has changed."""
    spec = models.resnet18_spec(6, image=64, classes=100)
    w, bound = models.synthetic_weights(spec, 46), models.SYNTHETIC_IMAGE_ABS_BOUND
    xs = [np.ascontiguousarray(models.synthetic_input(spec, 47 + i)) for i in range(4)]
    net, plain = (models.Network(spec, w, xs[0], input_abs_bound=bound, handover=h) for h in (True, False))
    feeder = models.HostFeeder(net, graph=graph)
    feeder.PART_BYTES = xs[0].nbytes // 3                                   # 2, 2, 2
    host = [torch.from_numpy(x).pin_memory() for x in xs]

    def expect(live=6):
        got = []
        plain.set_batch(live)
        for x in xs:
            plain.set_input(x[:live])
            got.append(plain.forward()[:live].clone())
        return got

    def run(on_result=lambda i: None):
        got = []
        def result(out):
            got.append(out.clone())
            on_result(len(got))
        feeder.run(host, result)
        return got

    assert len(feeder._cuts()) == 3
    first = expect()
    assert all(torch.equal(a, b) for a, b in zip(run(), first))
    old = [n.layers[5].bn_gpu for n in (net, plain)] + [net.layers[-1].output_gpu.detach()]
    for n in (net, plain):
        n.layers[5].bn_gpu = n.layers[5].bn_gpu + 9.0
    net.layers[-1].output_gpu.data = torch.zeros_like(net.layers[-1].output_gpu)
    second = expect()
    assert not torch.equal(first[0], second[0]) and len(old) == 3
    assert all(torch.equal(a, b) for a, b in zip(run(), second))
    four = expect(4)
    got = run(lambda i: net.set_batch(4) if i == 2 else None)
    assert all(torch.equal(a, b) for a, b in zip(got[:2], second[:2]))
    assert all(torch.equal(a[:4], b) for a, b in zip(got[2:], four[2:]))
    net.set_batch(6)
    assert all(torch.equal(a, b) for a, b in zip(run(), second)) and len(feeder.parts) == 3
    planes = [[l.input_planes for l in p.layers if getattr(l, "input_planes", None) is not None] for p in feeder.parts.values()]
    assert len(planes) == 3 and planes[0] and all(a is b for p in planes[1:] for a, b in zip(planes[0], p))


@pytest.mark.parametrize("which", ["resnet18", "vgg_cifar", "mlp"])
def test_set_batch_runs_ragged_batches_on_the_same_objects(cuda, which):
    """Layer objects built for 8 images process 5, then 8, then 3 images (Network.set_batch)
    without being rebuilt: every layer's bits and the logits of the live images equal the oracle's
    on exactly those images (the reference fixes the batch at construction, param.h:875-881)."""
    spec = {"resnet18": models.resnet18_spec(8, image=64, classes=100), "vgg_cifar": models.vgg_cifar_spec(8),
            "mlp": models.mlp_spec(8)}[which]
    w = models.synthetic_weights(spec, 80)
    bound = models.SYNTHETIC_IMAGE_ABS_BOUND if which == "resnet18" else None
    net = models.Network(spec, w, models.synthetic_input(spec, 81), input_abs_bound=bound)
    net.forward()
    for step, n in enumerate((5, 8, 3)):
        x = models.synthetic_input(spec, 90 + step, batch=n)
        net.set_batch(n)
        net.set_input(x)
        logits = (net.forward_graph() if step else net.forward())[:n].cpu().numpy()
        acts, ress = onet.run(dict(spec, batch=n), w, x)
        for i, (layer, a, r) in enumerate(zip(net.layers[:-1], acts[:-1], ress[:-1])):
            got = layer.get_output_gpu()[:n].cpu().numpy().view(np.uint32)
            assert np.array_equal(got.reshape(a.shape), a), "batch %d layer %d %s bits" % (n, i, layer.name)
            if r is not None:
                gr = layer.download_output_residual()
                assert np.array_equal(gr, r), "batch %d layer %d %s residual" % (n, i, layer.name)
        np.testing.assert_allclose(logits, acts[-1], rtol=1e-5, atol=1e-5)
    with pytest.raises(ValueError):
        net.set_batch(9)


@pytest.mark.parametrize("which,sub", [("mlp", 512), ("vgg_cifar", 32)])
def test_baseline_batch_logits_against_oracle_slice(cuda, which, sub):
    """The MLP at batch 8192 and the CIFAR VGG at batch 1024 (the standalone network
    configurations at their full batch): the logits of the first images must equal the CPU
    oracle's on exactly those images (every image is processed independently), and all logits
    must be finite.  1e-5 relative."""
    spec = models.mlp_spec(8192) if which == "mlp" else models.vgg_cifar_spec(1024)
    w = models.synthetic_weights(spec, 110)
    x = models.synthetic_input(spec, 111)
    net = models.Network(spec, w, x)
    logits = net.forward_graph().cpu().numpy()
    assert np.all(np.isfinite(logits))
    acts, _ = onet.run(dict(spec, batch=sub), w, x[:sub])
    np.testing.assert_allclose(logits[:sub], acts[-1], rtol=1e-5, atol=1e-5)
    # and the last images, which sit in the last tiles of every layer
    acts, _ = onet.run(dict(spec, batch=sub), w, x[-sub:])
    np.testing.assert_allclose(logits[-sub:], acts[-1], rtol=1e-5, atol=1e-5)
