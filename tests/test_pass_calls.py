"""What a network prepares for a pass, without a GPU: layer objects on CPU tensors, and a stand-in for the library that
records what it is asked."""
import ctypes as C

import pytest
import torch

from tcbnn_b200 import lib, models, ops, param


class _Library:
    def __init__(self):
        self.asked = []
        self.tcbnn_fc_chain_apart = lib.load().tcbnn_fc_chain_apart     # (asks no GPU)

    def tcbnn_fc_chain_fits(self, layers, n, M, K, ld):
        self.asked.append("fits")
        return int(64 <= M <= 960)

    def tcbnn_fc_chain_pays(self, widths, n, M):
        self.asked.append((list(widths), n, M))
        return int(64 <= M <= 960 and widths[n] < 1000)


@pytest.fixture
def library(monkeypatch):
    def need(*ts):
        for t in ts:
            if t is not None and not t.is_contiguous():
                raise lib.TcbnnError("contiguous")
    fake = _Library()
    models._one_launch_pays.cache_clear()
    monkeypatch.setattr(lib, "load", lambda: fake)
    monkeypatch.setattr(lib, "bound", lambda name: name)
    monkeypatch.setattr(ops, "_need_cuda", need)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    yield fake
    models._one_launch_pays.cache_clear()


def _ints(*shape):
    return torch.zeros(shape, dtype=torch.int32)


def _mlp(batch, widths):
    words = [ops.step128_words(n) for n in widths]
    first = param.In128LayerParam("Fin", batch, widths[0])
    first.input_gpu, first.output_gpu = torch.zeros((batch, widths[0])), _ints(batch, words[0])
    layers = [first]
    for i, (k, n) in enumerate(zip(widths, widths[1:])):
        last = i + 2 == len(widths)
        l = (param.Out128LayerParam if last else param.Fc128LayerParam)("L%d" % (i + 1), batch, k, n)
        l.weight_gpu, l.input_gpu, l.workspace = _ints(n, words[i]), layers[-1].output_gpu, None
        if last:
            l.bn_scale_gpu, l.bn_bias_gpu, l.output_gpu = torch.zeros(n), torch.zeros(n), torch.zeros((batch, n))
        else:
            l.bn_gpu, l.output_gpu = torch.zeros(n), _ints(batch, words[i + 1])
        layers.append(l)
    return layers


def _calls(layers):
    return models._Calls(layers).calls


def _names(layers):
    return [name for name, _ in _calls(layers)]


WIDTHS = (784, 1024, 512, 1024, 10)


def test_one_launch_follows_every_layers_input(library):
    """A layer's own input tensor counts where the whole pass is one call: given another storage in place, and where
    its rows do not lie one behind the other."""
    layers = _mlp(100, WIDTHS)
    assert _names(layers) == ["tcbnn_fc_chain"]
    layers[2].input_gpu = layers[1].output_gpu.view(100, -1)           # (a tensor of its own on the same rows)
    calls = models._Calls(layers)
    calls.note(layers)
    assert calls.hold(layers) and not calls.moved()
    layers[2].input_gpu.data = layers[2].input_gpu.clone()
    assert calls.moved() and "tcbnn_fc_chain" not in _names(layers)
    layers = _mlp(100, WIDTHS)
    wide = _ints(100, 2 * layers[1].output_gpu.shape[1])
    layers[1].output_gpu = layers[2].input_gpu = wide[:, :wide.shape[1] // 2]
    with pytest.raises(lib.TcbnnError):
        _calls(layers)


def _settled(layers):
    return [args[-1] for name, args in _calls(layers) if name in ("tcbnn_fc_layer_p", "tcbnn_out_layer_p")]


@pytest.mark.parametrize("which", ["weight_gpu", "bn_gpu", "bn_scale_gpu", "first"])
@pytest.mark.parametrize("batch", [8, 100, 2000])
def test_parameters_that_the_pass_writes_are_not_read_ahead(library, batch, which):
    """A layer whose weight or parameters lie in another layer's output has its launches one by one, and nothing is
    read or expanded before the layers in front have run."""
    widths = (256, 256, batch, 128, 10) if which == "weight_gpu" else (784, 1024, 512, 1024, 10)
    layers = _mlp(batch, widths)
    layers[0].expands = (layers[2],)
    layers[2].weight_units = layers[2].input_units = layers[1].next_units = torch.zeros(256, dtype=torch.uint8)
    before = _settled(layers)
    assert before == ([] if batch == 100 else [1] * 4)
    if which == "weight_gpu":                            # rows of activations against one another
        layers[2].weight_gpu = layers[1].output_gpu
    elif which == "bn_gpu":                              # (the last words of the buffer)
        layers[2].bn_gpu = layers[1].output_gpu.view(-1)[-512:].view(torch.float32) if batch > 8 else layers[1].output_gpu.view(torch.float32).view(-1)
    elif which == "bn_scale_gpu":
        layers[-1].bn_scale_gpu = layers[2].output_gpu.view(torch.float32).view(-1)[3:13]
    else:
        layers[1].weight_gpu = layers[0].output_gpu[-8:]
    assert _settled(layers) == [0] * 4
    for name, args in _calls(layers):
        if name == "tcbnn_pack_rows_w":
            assert args[-1] == 0                         # weights expanded at the start of the pass
        if name == "tcbnn_fc_layer_p":
            assert args[-4:-1] == (None, None, None)     # expanded operands
    layers = _mlp(batch, widths)                         # beside one another in one allocation is not within
    room = _ints(2 * layers[1].output_gpu.numel() + layers[2].weight_gpu.numel())
    n = layers[1].output_gpu.numel()
    layers[1].output_gpu = layers[2].input_gpu = room[:n].view(layers[1].output_gpu.shape)
    layers[2].weight_gpu = room[n:n + layers[2].weight_gpu.numel()].view(layers[2].weight_gpu.shape)
    assert _settled(layers) == before


@pytest.mark.parametrize("batch", [8, 2000])
def test_nothing_is_settled_behind_a_launch_that_need_not_wait(library, batch):
    """Only an input layer's launch waits for all before it: what a pass over later layers reads may still be written
    when its second launch starts."""
    layers = _mlp(batch, WIDTHS)
    assert _settled(layers) == [1] * 4
    assert _settled(layers[1:]) == [0] * 4
    assert _settled(layers[2:]) == [0] * 3
    layers[1].input_units = layers[1].weight_units = layers[2].weight_units = torch.zeros(256, dtype=torch.uint8)
    assert all(args[-4:-1] == (None, None, None) for name, args in _calls(layers[1:]) if name == "tcbnn_fc_layer_p")


def test_one_launch_only_on_buffers_of_their_own(library):
    """Rows are worked on at different times in one launch: an input that lies in a buffer of the pass, or two layers'
    outputs in one, need a launch after the other."""
    def chained(change):
        layers = _mlp(100, (512, 512, 512, 512, 512))
        change(layers)
        return _names(layers) == ["tcbnn_fc_chain"]

    def shared_output(layers):
        layers[3].output_gpu = layers[4].input_gpu = layers[1].output_gpu

    def input_is_output(layers):
        layers[0].input_gpu = layers[4].output_gpu

    def input_in_bits(layers):
        layers[0].input_gpu = torch.zeros(60000)[:51200].view(100, 512)
        layers[2].output_gpu = layers[3].input_gpu = layers[0].input_gpu.view(-1)[700:2300].view(torch.int32).view(100, 16)

    assert chained(lambda layers: None)
    assert not any(chained(f) for f in (shared_output, input_is_output, input_in_bits))
    # ... and an input that comes later
    layers = _mlp(100, (512, 512, 512, 512, 512))
    calls = models._Calls(layers)
    assert calls.serves(torch.zeros(100, 512)) and not calls.serves(layers[4].output_gpu)
    layers[0].input_gpu = layers[4].output_gpu
    other = models._Calls(layers)
    assert len(other.calls) == 5 and other.serves(layers[4].output_gpu)


class _Counted:
    """A layer that counts how often it is looked at."""

    def __init__(self, layer):
        self.__dict__.update(layer=layer, looks=0)

    def __getattr__(self, name):
        self.__dict__["looks"] += 1
        return getattr(self.layer, name)


@pytest.mark.parametrize("batch", [8, 100, 2000])
def test_another_input_tensor_costs_the_first_call_only(library, batch):
    """A pass on a tensor not seen before exchanges the input's address; nothing is prepared again, and no other layer
    looked at."""
    layers = _mlp(batch, WIDTHS)
    calls = models._Calls(layers)
    calls.note(layers)
    watched = layers[:1] + [_Counted(l) for l in layers[1:]]
    library.asked.clear()
    layers[0].input_gpu = x = torch.ones(batch, 784)
    p = models._Pass(calls, watched, fresh=False)
    assert not library.asked and not any(l.looks for l in watched[1:])
    assert p.calls[0][1][0] == x.data_ptr() and p.calls[1:] == calls.calls[1:]
    name, args = calls.calls[0]
    assert p.calls[0][0] == name and p.calls[0][1][1:4] == args[1:4]


@pytest.mark.parametrize("batch,widths", [(8, WIDTHS), (100, (784, 1000))])
def test_what_does_not_pay_in_one_launch_is_not_built(library, monkeypatch, batch, widths):
    """Passes that one launch would make slower, or cannot take, cost no list of layers."""
    def build(*a):
        raise AssertionError("built")
    layers = _mlp(batch, widths)
    monkeypatch.setattr(lib, "ChainLayer", build)
    assert _names(layers)[0] == "tcbnn_pack_rows_w"
    assert library.asked == ([] if batch == 8 else [(list(widths), len(widths) - 1, batch)])
