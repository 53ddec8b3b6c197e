"""The bit GEMM that reads packed rows (one launch) and the MLP that takes one launch, at the edges of their
tiles, against the CPU oracle and against the layers called one by one.  Integers and bits are exact; logits are
one fp32 multiply-add on an exact integer (rounded once here, twice in the oracle: 2^-23 of the larger term)."""
import numpy as np
import pytest
import torch

import oracle as orc
import util
from tcbnn_b200 import lib, models, ops

pytestmark = pytest.mark.gpu


def _dev(a, cuda):
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).to(cuda)


def _rows(words, ld, offset, cuda):
    """`words` on the GPU in rows of ld words that start `offset` words into an allocation."""
    t = torch.zeros((words.shape[0] * ld + offset,), dtype=torch.int32, device=cuda)[offset:].view(words.shape[0], ld)
    t[:, :words.shape[1]] = _dev(words, cuda)
    return t


# M, N, K; extra words per row, words in front of the first row.  As the library routes them: most of the small ones to the
# warp-level kernel.
SHAPES = [
    (1, 1, 1, 0, 0), (1, 10, 64, 0, 0), (31, 33, 65, 0, 0), (32, 128, 512, 0, 0), (33, 129, 513, 0, 0),
    (129, 200, 1000, 0, 0), (256, 128, 511, 0, 0), (257, 300, 449, 0, 0),
    (640, 4096, 200, 0, 0),            # packed rows: short K, several tiles per CTA
    (2000, 3000, 64, 0, 0),            # packed rows: one 64-bit block
    (5000, 1000, 1500, 0, 0),          # packed rows without scratch, integers
    (70, 130, 2112, 0, 0), (3, 1000, 16384, 0, 0),
    (40, 4096, 9216, 0, 0),            # packed rows: K cut over clusters
    (33, 140, 700, 4, 0), (33, 140, 700, 2, 0), (33, 140, 700, 0, 2), (300, 1100, 4100, 2, 2),
]


@pytest.mark.parametrize("M,N,K,pad,offset", SHAPES)
def test_gemm_family_on_packed_rows(cuda, M, N, K, pad, offset):
    g = util.rng(M + 3 * N + 7 * K)
    ld = orc.step128_words(K)
    A, W = (util.mask_row_pad(util.rand_words(g, (r, ld)), K) for r in (M, N))
    thr = (g.standard_normal(N) * np.sqrt(K)).astype(np.float32)
    thr[0] = np.nan                                                  # no value reaches it
    scale, bias = g.standard_normal(N).astype(np.float32), g.standard_normal(N).astype(np.float32)
    a, w = _rows(A, ld + pad, offset, cuda), _rows(W, ld + pad, offset, cuda)
    ref = orc.bgemm(A, W, K)
    ws = ops.gemm_workspace(M, N, K, cuda)
    got = ops.bgemm(a, w, K, workspace=ws)
    assert np.array_equal(got.cpu().numpy(), ref)
    assert torch.equal(got, ops.bgemm(a, w, K))                      # (and without scratch)
    bits = torch.full((M, orc.step128_words(N)), -1, dtype=torch.int32, device=cuda)
    ops.fc_layer(a, w, _dev(thr, cuda), K, out=bits, workspace=ws)
    words = (N + 31) // 32
    want = util.pm1_to_bits(np.where(ref >= thr, 1.0, -1.0))         # NaN: never
    assert np.array_equal(bits.cpu().numpy().view(np.uint32)[:, :words], want)
    assert (bits[:, words:] == -1).all()                             # nothing behind the last word is touched
    out = ops.out_layer(a, w, _dev(scale, cuda), _dev(bias, cuda), K, workspace=ws).cpu().numpy()
    exact = ref.astype(np.float64) * scale + bias
    np.testing.assert_allclose(out, exact, rtol=2.0 ** -23, atol=2.0 ** -23 * float(np.abs(bias).max()))
    assert ops.gemm_status() == 0


# Around one tile of every width, several tiles per CTA, and K of one bit, of one 64-bit block and one bit more, of whole
# stages of 512 bits and one bit less and more; then K cut over clusters: 8 stages of which the last is short, 16 of which
# the last has 20 bits, 18, which eight CTAs cannot share, 32.
TILES = [(1, 1, 1), (31, 33, 65), (32, 128, 512), (33, 129, 513), (97, 40, 64), (129, 200, 1000), (256, 128, 511), (257, 300, 449),
         (640, 4096, 200), (2000, 3000, 64), (2500, 1000, 1500), (70, 130, 4090), (300, 200, 7700), (40, 1100, 9216), (3, 1000, 16384)]


@pytest.mark.parametrize("M,N,K", TILES)
def test_every_tile_width_and_cluster_on_packed_rows(cuda, M, N, K):
    """The kernel on packed rows at every tile width and cluster size that K allows, in all three forms, its weight settled
    or not, and the next layer's expanded operand: against the oracle, and each time on this kernel."""
    g = util.rng(M + 3 * N + 7 * K + 1)
    ld = orc.step128_words(K)
    A, W = (util.mask_row_pad(util.rand_words(g, (r, ld)), K) for r in (M, N))
    thr = (g.standard_normal(N) * np.sqrt(K)).astype(np.float32)
    scale, bias = g.standard_normal(N).astype(np.float32), g.standard_normal(N).astype(np.float32)
    a, w, dthr, dscale, dbias = (_dev(t, cuda) for t in (A, W, thr, scale, bias))
    ref = orc.bgemm(A, W, K)
    exact = ref.astype(np.float64) * scale + bias
    close = dict(rtol=2.0 ** -23, atol=2.0 ** -23 * float(np.abs(bias).max()))
    words = orc.step128_words(N)
    signs = np.where(ref >= thr, 1.0, -1.0).astype(np.float32)
    want = torch.zeros((M, words), dtype=torch.int32, device=cuda)
    want[:, :(N + 31) // 32] = _dev(util.pm1_to_bits(signs), cuda)
    ref = torch.from_numpy(ref).to(cuda)
    # the next layer's operand, as the input layer lays it out
    units, packed = torch.zeros((-(-M // 128) * -(-N // 64) * 4096,), dtype=torch.uint8, device=cuda), torch.zeros_like(want)
    x = _dev(signs, cuda)
    lib.call("tcbnn_pack_rows_x", x.data_ptr(), M, N, words, packed.data_ptr(), units.data_ptr(), ops._stream())
    assert torch.equal(packed, want)
    stages, seen = -(-K // 512), set()
    try:
        ops.set_gemm_path(2)
        for cols in range(32, 257, 32):
            for splits in (1, 2, 4, 8):
                ops.set_gemm_bits_plan(cols, splits)
                fits = (splits - 1) * -(-stages // splits) < stages
                assert (ops.gemm_route(ops.GEMM_INT32, M, a, w, K, None) == ops.GEMM_ON_PACKED) == fits, (cols, splits)
                if not fits:
                    continue
                seen.add(splits)
                assert torch.equal(ops.bgemm(a, w, K), ref), (cols, splits)
                for settled in (0, 1):
                    bits, nxt = torch.zeros_like(want), torch.zeros_like(units)
                    lib.call("tcbnn_fc_layer_p", a.data_ptr(), w.data_ptr(), dthr.data_ptr(), M, K, N, ld, ld, bits.data_ptr(), words,
                             None, 0, None, None, nxt.data_ptr(), settled, ops._stream())
                    assert torch.equal(bits, want) and torch.equal(nxt, units), (cols, splits, settled)
                    out = torch.zeros((M, N), device=cuda)
                    lib.call("tcbnn_out_layer_p", a.data_ptr(), w.data_ptr(), dscale.data_ptr(), dbias.data_ptr(), M, K, N, ld, ld,
                             out.data_ptr(), N, None, 0, settled, ops._stream())
                    np.testing.assert_allclose(out.cpu().numpy(), exact, err_msg=str((cols, splits, settled)), **close)
        assert ops.gemm_status() == 0
        assert seen == {s for s in (1, 2, 4, 8) if (s - 1) * -(-stages // s) < stages}
    finally:
        ops.set_gemm_path(0)
        ops.set_gemm_bits_plan()


# extra words per row, words in front of the first row
@pytest.mark.parametrize("pad,offset,packed", [(0, 0, True), (4, 0, True), (0, 4, True), (2, 0, False), (0, 2, False), (2, 2, False)])
def test_rows_that_are_not_aligned_are_not_taken_packed(cuda, pad, offset, packed):
    """A shape that the library takes packed goes to another kernel where a row does not start on 16 bytes, also where packed
    rows are asked for: of either operand, with the same results."""
    M, N, K = 640, 2048, 200
    g = util.rng(5)
    ld = orc.step128_words(K)
    A, W = (util.mask_row_pad(util.rand_words(g, (r, ld)), K) for r in (M, N))
    ref = orc.bgemm(A, W, K)
    try:
        for path in (0, 2):
            ops.set_gemm_path(path)
            for which in (0, 1):
                a, w = (_rows(t, ld + (pad if i == which else 0), offset if i == which else 0, cuda) for i, t in enumerate((A, W)))
                assert (ops.gemm_route(ops.GEMM_INT32, M, a, w, K, None) == ops.GEMM_ON_PACKED) == packed
                assert np.array_equal(ops.bgemm(a, w, K).cpu().numpy(), ref)
    finally:
        ops.set_gemm_path(0)
    assert ops.gemm_status() == 0


def test_shapes_taken_packed_by_estimate(cuda):
    """Which of some shapes the library takes packed, so that a changed estimate shows."""
    for M, N, K, mode, room, route in [(640, 4096, 200, ops.GEMM_BITS, True, ops.GEMM_ON_PACKED), (2000, 3000, 64, ops.GEMM_INT32, True, ops.GEMM_ON_PACKED),
                                       (40, 4096, 9216, ops.GEMM_BITS, True, ops.GEMM_ON_PACKED), (1024, 1024, 4096, ops.GEMM_INT32, True, ops.GEMM_ON_PACKED),
                                       (1024, 512, 25088, ops.GEMM_BITS, True, ops.GEMM_ON_PACKED), (5000, 1000, 1500, ops.GEMM_INT32, False, ops.GEMM_ON_PACKED),
                                       (8, 1024, 1024, ops.GEMM_BITS, True, ops.GEMM_ON_B1), (33, 129, 513, ops.GEMM_BITS, True, ops.GEMM_ON_B1),
                                       (8192, 8192, 8192, ops.GEMM_INT32, True, ops.GEMM_ON_EXPANDED), (2048, 4096, 9216, ops.GEMM_BITS, True, ops.GEMM_ON_EXPANDED)]:
        ld = orc.step128_words(K)
        a, w = (torch.empty((r, ld), dtype=torch.int32, device=cuda) for r in (M, N))
        assert ops.gemm_route(mode, M, a, w, K, ops.gemm_workspace(M, N, K, cuda) if room else None) == route, (M, N, K)


def _graph_us(call, n=20):
    call()
    torch.cuda.synchronize()
    graph, best = torch.cuda.CUDAGraph(), 1e9
    with torch.cuda.stream(torch.cuda.Stream()):
        graph.capture_begin(capture_error_mode="thread_local")
        for _ in range(n):
            call()
        graph.capture_end()
    for _ in range(8):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end) * 1e3 / n)
    return best


def test_no_more_clusters_than_run_at_once(cuda):
    """K is cut over clusters only while all of them run at once: a second wave of a few (34 to 37 of four CTAs) doubled the
    call's time, 13.7 us where the kernel without clusters takes 9.8.  Within a quarter of that one now."""
    M, K = 18, 7364
    ld = orc.step128_words(K)
    for tiles in range(31, 38):
        N = 128 * tiles - 1
        a, w = (torch.zeros((r, ld), dtype=torch.int32, device=cuda) for r in (M, N))
        thr, out = torch.zeros(N, device=cuda), torch.zeros((M, orc.step128_words(N)), dtype=torch.int32, device=cuda)
        took = {}
        try:
            for path in (0, 3):
                ops.set_gemm_path(path)
                took[path] = _graph_us(lambda: ops.fc_layer(a, w, thr, K, out=out))
        finally:
            ops.set_gemm_path(0)
        assert took[0] < 1.25 * took[3], (tiles, took)


WIDTHS = [(784, 1024, 1024, 1024, 10), (100, 130, 1000, 64, 7), (1, 1, 1), (845, 1024, 928, 1000), (513, 40, 1024, 257, 1024),
          (1500, 96, 33, 500)]


@pytest.mark.parametrize("widths", WIDTHS)
@pytest.mark.parametrize("batch", [64, 65, 241, 300, 700])
def test_mlp_in_one_launch_is_its_layers_one_by_one(cuda, widths, batch):
    """Every layer's packed output and the logits of a pass in one launch, for 16, 32 and 64 rows per cluster with
    a ragged last one, against the same layers called by themselves; and of the network's own passes, which
    take the one launch or the layers' by what is faster."""
    spec = models.mlp_spec(batch, widths[0], 1, widths[-1])
    spec["layers"] = [spec["layers"][0]] + [dict(type="fc", name="Fc%d" % i, N=n) for i, n in enumerate(widths[1:-1])] + [spec["layers"][-1]]
    w, x = models.synthetic_weights(spec, 41), models.synthetic_input(spec, 42)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    assert models._chain_call(net.layers) is not None
    for l in plain.layers:
        l.forward()
    def one_launch():
        name, args, _ = models._chain_call(net.layers)
        lib.call(name, *args, ops._stream())
    for one_pass in [one_launch] + [net.forward] * 4:                # (a replayed graph by the last)
        for l in net.layers:
            l.output_gpu.fill_(0)
        one_pass()
        for l, p in zip(net.layers, plain.layers):
            assert torch.equal(l.output_gpu, p.output_gpu), l.name
    for fewer in (batch - 1, batch // 3):                            # in the same buffers; in one launch or, below 64 rows, in several
        net.set_batch(fewer)
        assert (models._chain_call(net.layers) is not None) == (fewer >= 64)
        for one_pass in ([one_launch] if fewer >= 64 else []) + [net.forward]:
            for l in net.layers:
                l.output_gpu.fill_(0)
            one_pass()
            for l, p in zip(net.layers, plain.layers):
                assert torch.equal(l.output_gpu[:fewer], p.output_gpu[:fewer]), l.name
                assert not l.output_gpu[fewer:].any()
    assert ops.gemm_status() == 0


@pytest.mark.parametrize("widths", [(784, 10), (784, 128, 10), (200, 1000), (784, 1024, 1000), (784, 1024, 1024, 1024, 10)])
def test_one_launch_is_not_taken_where_the_layers_are_faster(cuda, widths):
    """A pass takes no longer than its layers' launches, within a fifth: in one launch 784 -> 10 took 10.7 us on 700 rows where
    the two layers take 4.1."""
    for batch in (64, 200, 400, 700, 960):
        spec = models.mlp_spec(batch, widths[0], 1, widths[-1])
        spec["layers"] = [spec["layers"][0]] + [dict(type="fc", name="Fc%d" % i, N=n) for i, n in enumerate(widths[1:-1])] + [spec["layers"][-1]]
        net = models.Network(spec, models.synthetic_weights(spec, 73), models.synthetic_input(spec, 74))
        own = models._Pass(models._Calls(net.layers), net.layers)
        layers = [(lib.bound(name), args) for name, args, _ in (l._call_args(True) for l in net.layers)]

        def one_by_one():
            for f, args in layers:
                assert f(*args, ops._stream()) == 0
        took, theirs = _graph_us(own.run), _graph_us(one_by_one)
        assert took < 1.2 * theirs, (batch, took, theirs, own.common.chain)


def test_mlp_with_another_layers_input_is_not_one_launch(cuda):
    """A layer whose input is not the output of the one in front keeps its own launch, and its input counts."""
    spec = models.mlp_spec(72)
    w, x = models.synthetic_weights(spec, 43), models.synthetic_input(spec, 44)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    other = torch.randint(-2 ** 31, 2 ** 31, net.layers[2].input_gpu.shape, dtype=torch.int64, device=cuda).to(torch.int32)
    want = net.forward().clone()
    for n in (net, plain):
        n.layers[2].set_input_gpu(other.clone())
    assert models._chain_call(net.layers) is None
    for l in plain.layers:
        l.forward()
    got = net.forward().clone()
    assert torch.equal(got, plain.layers[-1].output_gpu) and not torch.equal(got, want)


@pytest.mark.parametrize("graph", [False, True])
def test_mlp_in_one_launch_follows_a_layers_input_given_another_storage(cuda, graph):
    """The rows of a layer's input tensor are exchanged in place, behind passes that are replayed by then."""
    spec = models.mlp_spec(200)
    w, x = models.synthetic_weights(spec, 47), models.synthetic_input(spec, 48)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    one_pass = net.forward_graph if graph else net.forward
    net.layers[2].input_gpu = net.layers[1].output_gpu.view(200, -1)
    for _ in range(4):
        want = one_pass().clone()
    assert models._Calls(net.layers).chain
    other = torch.randint(-2 ** 31, 2 ** 31, net.layers[2].input_gpu.shape, dtype=torch.int64, device=cuda).to(torch.int32)
    net.layers[2].input_gpu.data = other
    plain.layers[2].set_input_gpu(other)
    for l in plain.layers:
        l.forward()
    got = one_pass().clone()
    assert torch.equal(got, plain.layers[-1].output_gpu) and not torch.equal(got, want)


@pytest.mark.parametrize("which,batch", [("mlp", 8), ("mlp", 100), ("mlp", 1100), ("mlp", 2000), ("vgg_cifar", 70), ("resnet_cifar", 33)])
def test_launches_a_pass_makes(cuda, which, batch):
    """What a network says a pass launches, against the kernels in a graph of it."""
    spec = getattr(models, which + "_spec")(batch)
    net = models.Network(spec, models.synthetic_weights(spec, 71), models.synthetic_input(spec, 72))
    net.forward()
    assert len(util.kernels_launched(net.forward)) == net.kernel_launches()


def test_launches_a_call_makes(cuda):
    """What a layer says it launches, against the kernels in a graph of its call."""
    for M, N, K in [(32, 128, 256), (1024, 1000, 512), (2048, 4096, 9216), (200, 256, 200000)]:
        ld = orc.step128_words(K)
        a, w = (torch.zeros((r, ld), dtype=torch.int32, device=cuda) for r in (M, N))
        thr, out = torch.zeros(N, device=cuda), torch.zeros((M, orc.step128_words(N)), dtype=torch.int32, device=cuda)
        ws = ops.gemm_workspace(M, N, K, cuda)
        for room in (ws, None):
            ops.fc_layer(a, w, thr, K, out=out, workspace=room)
            seen = len(util.kernels_launched(lambda: ops.fc_layer(a, w, thr, K, out=out, workspace=room)))
            assert ops.gemm_call_launches(ops.GEMM_BITS, M, a, w, K, room) == seen, (M, N, K, room is None)
            assert seen <= ops.gemm_launches(M, N, K, room)


def test_mlp_entry_point_refuses_what_it_does_not_take(cuda):
    spec = models.mlp_spec(80)
    net = models.Network(spec, models.synthetic_weights(spec, 45), models.synthetic_input(spec, 46))
    name, (x, M, K, ld, bits, chain, n), _ = models._chain_call(net.layers)
    chain[1].N += 1                                                  # not the next layer's K
    assert not lib.load().tcbnn_fc_chain_fits(chain, n, M, K, ld)
    with pytest.raises(lib.TcbnnError):
        lib.call(name, x, M, K, ld, bits, chain, n, ops._stream())


@pytest.mark.parametrize("batch", [8, 100])
def test_small_mlp_follows_weights_and_parameters_written_between_passes(cuda, batch):
    """Layers of a pass read weights, thresholds, scale and bias ahead of the wait for the layer in front: what the
    library or torch writes into them right before a pass counts in it."""
    spec = models.mlp_spec(batch)
    w, other = models.synthetic_weights(spec, 31), models.synthetic_weights(spec, 33)
    x = models.synthetic_input(spec, 32)
    net, plain = models.Network(spec, w, x), models.Network(spec, other, x)
    for _ in range(4):
        net.forward()
    want = plain.forward().clone()
    assert not torch.equal(net.forward(), want)
    for n, p in zip(net.layers[1:], plain.layers[1:]):
        for name in ("weight_gpu", "bn_gpu", "bn_scale_gpu", "bn_bias_gpu"):
            if hasattr(n, name):
                getattr(n, name).copy_(getattr(p, name))
    assert torch.equal(net.forward(), want)
    g = util.rng(batch)
    src = torch.from_numpy(util.rand_words(g, (1024, 4)).view(np.int32)).to(cuda)
    big, zero = torch.zeros((1024, 4), dtype=torch.int32, device=cuda), torch.zeros(1024, device=cuda)
    for _ in range(3):                                   # the library's own launch in front of the pass
        ops.fc_layer(src, big, zero, 128, out=net.layers[2].weight_gpu)
        got = net.forward().clone()
        plain.layers[2].weight_gpu.copy_(net.layers[2].weight_gpu)
        assert torch.equal(got, plain.forward())
        src.bitwise_not_()


@pytest.mark.parametrize("batch", [8, 100, 1024])
def test_a_layers_output_as_the_next_ones_weight(cuda, batch):
    """Rows of activations against one another: the weight is what the same pass has just computed, whichever launches
    the pass would take otherwise."""
    spec = models.mlp_spec(batch)
    spec["layers"][2] = dict(type="fc", name="Fc2", N=batch)
    w = models.synthetic_weights(spec, 51)
    inputs = [torch.from_numpy(models.synthetic_input(spec, s)).to(cuda) for s in (52, 53)]
    net, plain = (models.Network(spec, w, inputs[0], handover=h) for h in (True, False))
    for n in (net, plain):
        n.layers[2].weight_gpu = n.layers[1].output_gpu
    for i in (0, 1, 0, 0, 0, 1):
        net.layers[0].input_gpu = plain.layers[0].input_gpu = inputs[i]
        for l in plain.layers:
            l.forward()
        got = net.forward()
        for l, p in zip(net.layers, plain.layers):
            assert torch.equal(l.output_gpu, p.output_gpu), l.name
        assert torch.equal(got, plain.layers[-1].output_gpu)
    assert ops.gemm_status() == 0


@pytest.mark.parametrize("batch,live", [(1100, 1100), (1400, 1100), (1400, 1400)])
def test_operands_are_expanded_for_layers_that_read_them(cuda, batch, live):
    """In a pass, a layer's operands are laid out expanded where its call takes the kernel that reads them so, and
    nowhere else."""
    spec = models.mlp_spec(batch)
    w, x = models.synthetic_weights(spec, 61), models.synthetic_input(spec, 62)
    net, plain = models.Network(spec, w, x), models.Network(spec, w, x, handover=False)
    net.set_batch(live)
    for prod, l in list(zip(net.layers, net.layers[1:-1]))[live == 1100:]:       # (784 x 1024 is too small at 1100)
        route = ops.gemm_route(ops.GEMM_BITS, live, l.input_gpu, l.weight_gpu, l.input_width, l.workspace, True, True)
        assert route == (ops.GEMM_ON_PACKED if live == 1100 else ops.GEMM_ON_EXPANDED)
        expanded = route == ops.GEMM_ON_EXPANDED
        assert l.reads_units == (l in net.layers[0].expands) == expanded, l.name
        assert (l.input_units is not None) == (prod.next_units is not None) == expanded
        assert all((u is not None) == expanded for u in l._call_args(True)[1][-4:-2])
    for l in plain.layers:
        l.forward()
    for _ in range(4):
        assert torch.equal(net.forward()[:live], plain.layers[-1].output_gpu[:live])
