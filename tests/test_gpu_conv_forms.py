"""Forms that a convolution's launches take by size and alignment, at their edges, against the CPU oracle (bits,
integers and fp32 sums are exact)."""
import numpy as np
import pytest
import torch

import oracle as orc
import util
from tcbnn_b200 import ops

pytestmark = pytest.mark.gpu


def _dev(a, cuda):
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).to(cuda)


def _u32(t):
    return t.cpu().numpy().view(np.uint32)


# B, H, W, C, O, stride, pool; words in front of the input (the expansion pass takes four words of a pixel where they are
# 16-byte aligned, two otherwise; the pooling pass one, two or four words of a pixel by their number)
FORMS = [
    (2, 7, 9, 64, 64, 1, 1, 0), (2, 7, 9, 128, 64, 1, 1, 0), (2, 7, 9, 128, 64, 1, 1, 2), (3, 8, 6, 192, 64, 1, 1, 0),
    (3, 8, 6, 256, 32, 2, 1, 0), (3, 8, 6, 256, 32, 2, 1, 2), (1, 1, 1, 128, 128, 1, 1, 0),
    (2, 10, 6, 64, 32, 1, 2, 0), (2, 10, 6, 64, 96, 1, 2, 0), (2, 10, 6, 64, 128, 1, 2, 0), (40, 160, 160, 64, 64, 1, 2, 0),
    (160, 64, 64, 64, 128, 1, 2, 0),
]


@pytest.mark.parametrize("form", FORMS)
def test_expansion_and_pooling_passes(cuda, form):
    B, H, W, C, O, st, pool, front = form
    g = util.rng(sum(form))
    x = util.rand_words(g, (B, H, W, C // 32))
    f = util.rand_words(g, (O, 9, C // 32))
    thr = (g.standard_normal(O) * np.sqrt(C * 9) * 0.5).astype(np.float32)
    d = ops.conv_desc(B, H, W, C, O, 3, 3, st, st, True, pool)
    room = torch.zeros((x.size + front,), dtype=torch.int32, device=cuda)
    dx = room[front:].view(x.shape)
    dx.copy_(_dev(x, cuda))
    prep = ops.conv_prepare(d, _dev(f, cuda))
    go, _, _ = ops.conv_layer(d, dx, prep, _dev(thr, cuda))
    assert ops.conv_status(d, prep) == 0
    n = min(B, 3)                                        # (the oracle on the first and the last images)
    for part in {(0, n), (B - n, B)}:
        eo, _, _ = orc.conv_layer(x[part[0]:part[1]], f, thr, C, 3, 3, st, st, True, pool)
        assert np.array_equal(_u32(go)[part[0]:part[1]].reshape(eo.shape), eo), part


# R, S, O: one tap, two, three; channels that share their first two terms, and a filter all of whose channels do
@pytest.mark.parametrize("R,S,O,same", [(1, 1, 40, False), (1, 2, 64, False), (2, 1, 5, False), (1, 3, 70, False), (3, 3, 64, True), (3, 3, 96, False)])
def test_first_layer_sums_of_few_taps(cuda, R, S, O, same):
    """The compiled first layer makes its sums from the first two taps, shared between channels that agree in them:
    sums, residuals and bits of the oracle, with zeros among the pixels (a sum of -0 is stored as 0)."""
    g = util.rng(R * 100 + S * 10 + O)
    B, H, W = 3, 13, 11
    x = g.standard_normal((B, 3, H, W)).astype(np.float32)
    x[:, :, :4] = 0.0
    F = g.standard_normal((R * S, 3, O)).astype(np.float32)
    if same:
        F[:2] = F[:2, :, :1]
    thr = (g.standard_normal(O) * 2).astype(np.float32)
    thr[0] = 0.0
    eo, er, ea = orc.inconv_layer(x, F, thr, R, S, 1, 1, True, 1, save_residual=True, want_acc=True)
    d = ops.conv_desc(B, H, W, 3, O, R, S, 1, 1, True, 1)
    fb = ops.pack_inconv_filter(_dev(F, cuda))
    spec = ops.inconv_specialize(d, fb, _dev(thr, cuda))
    go, gr, ga = ops.inconv_layer(d, _dev(x, cuda), fb, _dev(thr, cuda), save_residual=True, want_acc=True, specialized=spec)
    assert np.array_equal(ga.cpu().numpy().view(np.uint32), ea.view(np.uint32))        # (the sign of a zero too)
    assert np.array_equal(gr.cpu().numpy(), er)
    assert np.array_equal(_u32(go), eo)
    spec.release()


def _check_pairs(cuda, form, images, pairs=True):
    """A layer three times in a row, compared with the oracle on ranges of its images; pairs: whether it runs on pairs
    of SMs."""
    B, H, W, C, O, rin, rout = form
    g = util.rng(B + H + W + C + O)
    x = util.rand_words(g, (B, H, W, C // 32))
    f = util.rand_words(g, (O, 9, C // 32))
    thr = (g.standard_normal(O) * np.sqrt(C * 9) * 0.5).astype(np.float32)
    pooled = rin is not None and rin.startswith("pooled")
    kind = rin.replace("pooled ", "") if rin not in (None, "acc") else None
    rc = 256 if pooled else O                            # a pooled residual goes into the first channels
    res = dres = None
    if kind:
        res = g.integers(-1500, 1501, size=(B, H * (2 if pooled else 1), W * (2 if pooled else 1), rc)).astype(np.int32)
        dres = torch.from_numpy(res).to(cuda)
        if kind != "int32":
            dres = dres.to(torch.int16)
        if kind == "chunked":
            dres = ops.nhwc_to_chunked(dres)
    d = ops.conv_desc(B, H, W, C, O, 3, 3)
    prep = ops.conv_prepare(d, _dev(f, cuda))
    dx, dthr = _dev(x, cuda), _dev(thr, cuda)

    def call():
        return ops.conv_layer(d, dx, prep, dthr, res_in=dres, residual_channels=rc if kind else 0, residual_pool=pooled,
                              save_residual=rout is not None, want_acc=rin == "acc",
                              residual_dtype=torch.int32 if rout == "int32" else torch.int16,
                              res_in_chunked=kind == "chunked", res_out_chunked=rout == "chunked")

    expect = {(lo, hi): orc.conv_layer(x[lo:hi], f, thr, C, 3, 3, 1, 1, True, 1, res_in=None if res is None else res[lo:hi],
                                       residual_channels=rc if kind else 0, residual_pool=pooled, save_residual=rout is not None,
                                       want_acc=rin == "acc") for lo, hi in images}
    for _ in range(3):
        go, gr, ga = call()
        assert ops.conv_status(d, prep) == 0
        if rout == "chunked":
            gr = ops.chunked_to_nhwc(gr)
        for (lo, hi), (eo, er, ea) in expect.items():
            assert np.array_equal(_u32(go[lo:hi]).reshape(eo.shape), eo), (lo, hi)
            if rout is not None:
                assert np.array_equal(gr[lo:hi].cpu().numpy().astype(np.int32), er), (lo, hi)
            if rin == "acc":
                assert np.array_equal(ga[lo:hi].cpu().numpy(), ea), (lo, hi)
    assert any("k_conv_umma_pair" in name for name in util.kernels_launched(call)) == pairs


# B, H, W, C, O, residual in / out.  3x3 layers of more than 256 channels run on pairs of SMs from two tiles per CTA on, with
# residuals or sums from two tiles per pair.  Here a pair has one tile or none: odd numbers of tiles (a pair whose second
# CTA has none), one block per stage.
PAIR_FORMS = [
    (29, 8, 8, 512, 512, None, None), (121, 7, 7, 512, 256, None, None), (121, 8, 8, 384, 128, None, None), (30, 8, 9, 448, 512, None, None),
    (29, 8, 8, 512, 512, "int16", "int16"), (33, 8, 8, 512, 512, "int32", "int32"), (29, 8, 8, 512, 512, None, "int32"),
    (31, 8, 8, 512, 512, "chunked", "chunked"), (31, 8, 8, 512, 512, None, "chunked"), (60, 6, 8, 512, 512, "pooled chunked", "chunked"),
    (60, 6, 8, 512, 512, "pooled int32", "int32"), (29, 8, 8, 512, 512, "acc", None),
]


@pytest.mark.parametrize("form", PAIR_FORMS)
def test_wide_layers_on_pairs_of_sms(cuda, form):
    _check_pairs(cuda, form, [(0, form[0])], pairs=form[5] is None and form[6] is None)


# Four or five tiles per pair and an odd number in all (159, 633, 635): both epilogue groups, accumulators handed back to the
# leader and used again, for each form of epilogue.  Images of 56 pixels a row have the longest second copy (NPOS 248).
PAIR_RUNS = [
    (251, 8, 8, 512, 512, None, None), (1000, 8, 8, 384, 128, None, None), (25, 56, 56, 384, 128, None, None),
    (251, 8, 8, 512, 512, "int16", "int16"), (251, 8, 8, 512, 512, "int32", "int32"), (251, 8, 8, 512, 512, None, "int16"),
    (251, 8, 8, 512, 512, None, "int32"), (251, 8, 8, 512, 512, "chunked", "chunked"), (251, 8, 8, 512, 512, None, "chunked"),
    (323, 6, 8, 512, 512, "pooled chunked", "chunked"), (251, 8, 8, 512, 512, "acc", None), (323, 6, 8, 512, 512, "pooled int32", "int32"),
]


@pytest.mark.parametrize("form", PAIR_RUNS)
def test_wide_layers_with_several_tiles_per_pair(cuda, form):
    B = form[0]
    n = 1 if B < 50 else 4
    _check_pairs(cuda, form, [(0, n), (B // 3, B // 3 + n), (B // 2, B // 2 + n), (B - n, B)], pairs=form[5] != "pooled int32")
