"""The torch.library operator kudnn_b200::linear and the nn.Linear drop-in module (kudnn_b200/torch_ops.py): the
documented PyTorch integration point of the reference (docs/zh/KuDNN_development_guide.md:1748-1775) on this side."""
import collections
import types

import numpy as np
import pytest
import torch

import kudnn_b200 as kb
from kudnn_b200 import torch_ops
from oracle import ko
from tests import helpers


def test_fake_implementation_propagates_shapes_without_a_device():
    x = torch.empty(3, 7, 64, dtype=torch.bfloat16, device="meta")
    w = torch.empty(96, 64, dtype=torch.bfloat16, device="meta")
    b = torch.empty(96, dtype=torch.bfloat16, device="meta")
    y = torch.ops.kudnn_b200.linear(x, w, b, kb.ACT_SWISH)
    assert y.shape == (3, 7, 96) and y.dtype == torch.bfloat16 and y.device.type == "meta"
    r = torch.empty(3, 7, 96, dtype=torch.bfloat16, device="meta")
    assert torch.ops.kudnn_b200.linear(x, w, None, 0, 1.0, r, kb.RES_IDENTICAL).shape == (3, 7, 96)


class _RecordedLinear:
    """Stands in for a primitive: remembers the weights it packed."""

    def __init__(self, desc):
        self.closed, self.graphs = False, 0

    def prepack(self, b, stream=None):
        self.weights = b.clone()

    def close(self):
        self.closed = True


@pytest.fixture
def recorded_handles(monkeypatch):
    monkeypatch.setattr(torch_ops.capi, "Linear", _RecordedLinear)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=1))
    monkeypatch.setattr(torch_ops, "_HANDLES", collections.OrderedDict())

    def handle(weight, m=4):
        x = torch.zeros(m, weight.shape[1])
        return torch_ops._handle(m, weight.shape[0], weight.shape[1], x, weight, None, 0, 1.0, None, 0)

    return handle


def test_weights_where_freed_ones_were_are_packed_again(recorded_handles):
    memory = np.zeros((8, 16), dtype=np.float32)
    first = torch.from_numpy(memory)
    old = recorded_handles(first)
    assert recorded_handles(first) is old and recorded_handles(first[:]) is old
    where = first.data_ptr()
    del first
    memory[:] = 1.0
    second = torch.from_numpy(memory)
    assert second.data_ptr() == where and second._version == 0
    assert torch.equal(recorded_handles(second).weights, second)
    second.add_(1.0)
    assert torch.equal(recorded_handles(second).weights, second)


def test_a_full_cache_keeps_primitives_that_graphs_use(recorded_handles, monkeypatch):
    monkeypatch.setattr(torch_ops, "_MAX_HANDLES", 3)
    weight = torch.zeros(8, 16)
    first = [recorded_handles(weight, m) for m in (1, 2, 3)]
    first[0].graphs = 1
    fourth = recorded_handles(weight, 4)
    assert [recorded_handles(weight, m) for m in (1, 3, 4)] == [first[0], first[2], fourth]
    assert not any(lin.closed for lin in first)  # a caller may be about to run the one that was dropped
    assert recorded_handles(weight, 2) is not first[1]


def _oracle(x, w, b, act, res, res_op):
    code = {torch.float32: kb.F32, torch.float16: kb.F16, torch.bfloat16: kb.BF16}[x.dtype]
    m, k = x.reshape(-1, x.shape[-1]).shape
    n = w.shape[0]
    desc = kb.make_desc(m, n, k, code, has_bias=b is not None, act=act, res_op=res_op)

    def st(t):
        t = t.detach().cpu().contiguous()
        return t.numpy() if t.dtype == torch.float32 else t.view(torch.int16).numpy().view(np.uint16)
    c = np.zeros((m, n), dtype=ko.np_dtype(code))
    o = np.zeros((m, n), dtype=ko.np_dtype(code)) if res_op else None
    ko.linear(helpers.oracle_desc(desc), st(x.reshape(m, k)), st(w), c, st(b) if b is not None else None,
              st(res.reshape(m, n)) if res is not None else None, o)
    return (o if res_op else c), code, st


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_linear_silu_module_matches_the_oracle(cuda_device, dtype):
    torch.manual_seed(5)
    layer = torch.nn.Linear(512, 1024, bias=True, device=cuda_device, dtype=dtype)
    with torch.no_grad():
        layer.weight.mul_(0.5)
    mod = torch_ops.Linear.from_torch(layer, act="silu")
    x = torch.randn(4, 50, 512, device=cuda_device, dtype=dtype)
    with torch.no_grad():
        y = mod(x)
    assert y.shape == (4, 50, 1024)
    ref, code, st = _oracle(x, layer.weight, layer.bias, kb.ACT_SWISH, None, kb.RES_NONE)
    helpers.compare(st(y.reshape(200, 1024)), ref, code)
    # decode shape with a gate operand, and weights updated in place (a fresh primitive packs the new values)
    gate = torch.randn(2, 1024, device=cuda_device, dtype=dtype)
    mul = torch_ops.Linear.from_torch(layer, residual="mul")
    with torch.no_grad():
        layer.weight.add_(0.01)
        y2 = mul(x[0, :2], gate)
    ref2, code, st = _oracle(x[0, :2], layer.weight, layer.bias, kb.ACT_NONE, gate, kb.RES_ELTWISE_MUL)
    helpers.compare(st(y2), ref2, code)
    torch_ops.clear_cache()


@pytest.mark.gpu
def test_operator_passes_opcheck(cuda_device):
    x = torch.randn(6, 64, device=cuda_device, dtype=torch.bfloat16)
    w = torch.randn(48, 64, device=cuda_device, dtype=torch.bfloat16)
    b = torch.randn(48, device=cuda_device, dtype=torch.bfloat16)
    torch.library.opcheck(torch.ops.kudnn_b200.linear.default, (x, w, b, kb.ACT_RELU, 0.0),
                          test_utils=("test_schema", "test_faketensor"))
    torch_ops.clear_cache()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,dtype", [(200, 520, 1024, torch.float32), (1, 700, 4104, torch.bfloat16), (4, 1003, 6152, torch.bfloat16),
                                         (60, 512, 1030, torch.float16)])
def test_one_layer_on_two_streams_and_in_graphs(cuda_device, m, n, k, dtype):
    """Scratch (split activations, partial sums and counters, packed rows) is written by every call; calls on different
    streams and replays of different graphs overlap."""
    torch.manual_seed(11)
    mod = torch_ops.Linear.from_torch(torch.nn.Linear(k, n, device=cuda_device, dtype=dtype), act="silu")
    xs = [torch.randn(m, k, device=cuda_device, dtype=dtype) for _ in range(4)]
    with torch.no_grad():
        want = [mod(x) for x in xs]
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in range(4)]
        outs = [[], [], [], []]
        for _ in range(40):
            for i in range(2):
                with torch.cuda.stream(streams[i]):
                    outs[i].append(mod(xs[i]))
        torch.cuda.synchronize()
        graphs = []
        for i in (2, 3):
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1]):
                outs[i] += [mod(xs[i]) for _ in range(8)]
        for out in outs[2] + outs[3]:
            out.zero_()
        torch.cuda.synchronize()
        for _ in range(10):
            for i in range(4):
                with torch.cuda.stream(streams[i]):
                    graphs[i - 2].replay() if i >= 2 else outs[i].append(mod(xs[i]))
        torch.cuda.synchronize()
    for got, ref in zip(outs, want):
        assert all(torch.equal(y, ref) for y in got)
    (lin, _), = torch_ops._HANDLES.values()
    assert lin.graphs == 2
    del graphs
    torch.cuda.synchronize()
    torch_ops.clear_cache()
