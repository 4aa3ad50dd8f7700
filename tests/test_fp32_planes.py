"""fp32 products as planes of fp16: the error bound of the split over tile edges, and rows that the planes do not carry, which the
device sends to the TF32 form, also in a captured graph."""
import pytest
import torch

import kudnn_b200 as kb

pytestmark = pytest.mark.gpu

_ACTS = {kb.ACT_NONE: lambda v: v, kb.ACT_RELU: torch.relu, kb.ACT_SWISH: torch.nn.functional.silu,
         kb.ACT_GELU_TANH: lambda v: torch.nn.functional.gelu(v, approximate="tanh")}


def _layer(monkeypatch, planes, m, n, k, w, owned=False, **desc):
    monkeypatch.setenv("KUDNN_B200_TC_PLANES", planes)
    lin = kb.Linear(kb.make_desc(m, n, k, kb.F32, b_strides=(n, 1) if owned else None, **desc))
    lin.force_kernel(kb.KERNEL_TC)
    lin.prepack(w, stream=torch.cuda.current_stream().cuda_stream)
    return lin


def _draw(device, *shape):
    gen = torch.Generator(device=device)
    gen.manual_seed(sum(shape))
    return torch.randn(shape, generator=gen, device=device)


@pytest.mark.parametrize("m,n,k,owned", [(1, 4, 8, False), (255, 260, 64, True), (257, 128, 68, False), (300, 1032, 1100, True), (2600, 1028, 72, False),
                                         (130, 300, 8200, False), (1024, 2500, 704, True), (300, 1030, 640, False)])
@pytest.mark.parametrize("act,bias,alpha", [(kb.ACT_NONE, False, 1.0), (kb.ACT_RELU, True, 1.0), (kb.ACT_SWISH, True, 0.5), (kb.ACT_GELU_TANH, False, 1.0)])
def test_error_of_the_planes(cuda_device, monkeypatch, m, n, k, owned, act, bias, alpha):
    stream = torch.cuda.current_stream().cuda_stream
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, *((k, n) if owned else (n, k))) * 0.02
    # rows of very different size, and one of zeros: each has its own scale
    a *= torch.pow(2.0, torch.randint(-40, 20, (m, 1), device=cuda_device)).float()
    a[m // 2] = 0.0
    side = _draw(cuda_device, n) if bias else None
    pitch = (n + 3) // 4 * 4 + 4
    lin = _layer(monkeypatch, "1", m, n, k, w, owned, has_bias=bias, act=act, act_alpha=0.0 if act == kb.ACT_RELU else 1.0, c_strides=(pitch, 1))
    c = torch.full((m, pitch), 7.0, device=cuda_device)
    for _ in range(2):
        lin.run(a, w, c, side, alpha=alpha, stream=stream)
    lin.check(stream=stream)
    assert lin.last_launches == (4 if n % 4 == 0 else 2)  # rows that end inside 16 bytes stay on the TF32 planes
    w64 = w.double() if owned else w.double().T
    pre = alpha * (a.double() @ w64) + (side.double() if bias else 0.0)
    want = _ACTS[act](pre)
    # each operand is carried to 2^-22, the product of the low parts (2^-22) is left out, and k / 16 additions to an accumulator, three
    # per step, each cut at 2^-23 of a partial sum; the activations' slope is at most 1.13
    size = alpha * (a.double().abs() @ w64.abs()) + (side.double().abs() if bias else 0.0)
    bound = 1.13 * (3 * 2.0 ** -22 + (k / 16 * 3 + 4) * 2.0 ** -23) * size + 2.0 ** -22 * want.abs()
    assert bool(((c[:, :n].double() - want).abs() <= bound).all())
    assert bool((c[:, n:] == 7.0).all())


@pytest.mark.parametrize("where,value", [((0, 0), float("inf")), ((3, 5), 1e-20), ((699, 999), float("nan")), ((5, 7), 1e30), ((699, slice(None)), 1e-40)])
def test_rows_the_planes_do_not_carry(cuda_device, monkeypatch, where, value):
    m, n, k = 700, 1000, 1000
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    marked = a.clone()
    marked[where] = value
    want = []
    planes, tf32 = (_layer(monkeypatch, p, m, n, k, w) for p in "10")
    for x in (a, marked):
        c = torch.empty((m, n), device=cuda_device)
        tf32.run(x, w, c, stream=torch.cuda.current_stream().cuda_stream)
        want.append(c)
    c, x = torch.empty((m, n), device=cuda_device), a.clone()
    planes.run(x, w, c, stream=torch.cuda.current_stream().cuda_stream)  # scratch exists before the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        planes.run(x, w, c, stream=torch.cuda.current_stream().cuda_stream)
    for source, ref, exact in ((a, want[0], False), (marked, want[1], True), (a, want[0], False)):
        x.copy_(source)
        graph.replay()
        torch.cuda.synchronize()
        # the same launches on the TF32 planes, bit by bit; or two forms, each within 2^-20 (|a| |w|)
        if exact:
            assert torch.equal(c.nan_to_num(1.5), ref.nan_to_num(1.5))
        else:
            assert bool(((c - ref).abs() <= 2.0 ** -16 * (source.abs() @ w.abs().T)).all()) and not torch.equal(c, ref)
    assert planes.last_launches == 4 and tf32.last_launches == 2
    planes.check()


@pytest.mark.parametrize("value", [float("inf"), 1e-25, 1e25])
def test_weights_the_planes_do_not_carry(cuda_device, monkeypatch, value):
    m, n, k = 300, 520, 328
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    w[519, 327] = value
    outs = []
    for planes in "01":
        lin = _layer(monkeypatch, planes, m, n, k, w)
        outs.append(torch.empty((m, n), device=cuda_device))
        lin.run(a, w, outs[-1], stream=torch.cuda.current_stream().cuda_stream)
        lin.check()
        assert lin.last_launches == 2
    assert torch.equal(outs[0].nan_to_num(1.5), outs[1].nan_to_num(1.5))


def test_a_pre_pack_that_fails_leaves_no_copy_under_the_old_pointer(cuda_device, monkeypatch):
    m, n, k = 300, 520, 328
    a, marked, plain = _draw(cuda_device, m, k), _draw(cuda_device, n, k), _draw(cuda_device, n, k + 1)[:, :k].contiguous()
    marked[519, 327] = 1e-25
    stream = torch.cuda.current_stream().cuda_stream
    want = {}
    for w in (marked, plain):
        want[w] = torch.empty((m, n), device=cuda_device)
        _layer(monkeypatch, "0", m, n, k, w).run(a, w, want[w], stream=stream)
    lin = _layer(monkeypatch, "1", m, n, k, marked)
    try:
        kb.debug_fail_allocation(0)
        lin.prepack(plain, stream=stream)
    except kb.KudnnError as err:
        assert err.status == 3
    finally:
        kb.debug_fail_allocation(-1)
    for w in (marked, plain):
        c = torch.empty((m, n), device=cuda_device)
        lin.run(a, w, c, stream=stream)
        lin.check()
        assert bool(((c - want[w]).abs() <= 2.0 ** -16 * (a.abs() @ w.abs().T)).all())


@pytest.mark.parametrize("where", ["weights", "activations"])
def test_without_memory_for_the_planes_the_call_takes_the_tf32_form(cuda_device, monkeypatch, where):
    m, n, k = 300, 520, 328
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    stream = torch.cuda.current_stream().cuda_stream
    want, c = (torch.empty((m, n), device=cuda_device) for _ in range(2))
    _layer(monkeypatch, "0", m, n, k, w).run(a, w, want, stream=stream)
    monkeypatch.setenv("KUDNN_B200_TC_PLANES", "1")
    lin = kb.Linear(kb.make_desc(m, n, k, kb.F32))
    lin.force_kernel(kb.KERNEL_TC)
    try:
        if where == "weights":
            kb.debug_fail_allocation(1)  # the status block, both kinds of planes together, the TF32 planes alone
        lin.prepack(w, stream=stream)
        if where != "weights":
            kb.debug_fail_allocation(1)  # one allocation for both kinds of planes, and no other
        lin.run(a, w, c, stream=stream)
    finally:
        kb.debug_fail_allocation(-1)
    lin.check()
    assert bool(((c - want).abs() <= 2.0 ** -16 * (a.abs() @ w.abs().T)).all())
    # and with memory again, the planes
    lin.prepack(w, stream=stream)
    lin.run(a, w, c, stream=stream)
    lin.check()
    assert lin.last_launches == 4 and bool(((c - want).abs() <= 2.0 ** -16 * (a.abs() @ w.abs().T)).all())


def test_graphs_follow_weights_that_are_pre_packed_again(cuda_device, monkeypatch):
    """A captured launch on the planes, replayed after the weights changed in place and were pre-packed again: to rows that the
    planes do not carry, and back."""
    m, n, k = 300, 520, 328
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    stream = torch.cuda.current_stream().cuda_stream
    lin = _layer(monkeypatch, "1", m, n, k, w)
    c, other, want = (torch.empty((m, n), device=cuda_device) for _ in range(3))
    lin.run(a, w, c, stream=stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lin.run(a, w, c, stream=torch.cuda.current_stream().cuda_stream)
    first = w.clone()
    second = _draw(cuda_device, n, k + 1)[:, :k].contiguous()
    for source, value in ((first, None), (second, 1e-25), (second, None), (first, 1e30), (first, None)):
        w.copy_(source)
        if value is not None:
            w[519, 327] = value
        lin.prepack(w, stream=stream)
        graph.replay()
        lin.run(a, w, other, stream=stream)
        lin.check()
        _layer(monkeypatch, "0", m, n, k, w).run(a, w, want, stream=stream)
        monkeypatch.setenv("KUDNN_B200_TC_PLANES", "1")
        for got in (c, other):
            assert bool(((got - want).abs() <= 2.0 ** -16 * (a.abs() @ w.abs().T)).all())


def _tail(a, w, form, low):
    """Every row has one large element that meets zeros, and otherwise only elements of about 2^low of it: `few` of them (the rest
    of the row zero), or all of the columns."""
    k = a.shape[1]
    a, w = a.clamp(-3.0, 3.0), w.clone()
    sign = torch.where(a < 0.0, -1.0, 1.0)
    small = sign * (1.0 + 0.9 * torch.rand_like(a)) * 2.0 ** low
    if form == "few":
        at = (torch.arange(a.shape[0], device=a.device)[:, None] * 37 + torch.tensor([3, 64, 65, 127, k - 1], device=a.device)) % (k - 2) + 2
        small = torch.zeros_like(small).scatter(1, at, small.gather(1, at))
    small[:, :2] = 0.0
    small[:, 0] = 1.0
    w[:, 0] = 0.0
    return small, w


@pytest.mark.parametrize("low", [-27, -28, -29, -30, -31, -32, -33, -34])
@pytest.mark.parametrize("form", ["few", "all"])
@pytest.mark.parametrize("operand", ["activations", "weights"])
def test_small_elements_of_a_row_keep_their_bits(cuda_device, monkeypatch, low, form, operand):
    """Results that only elements far below their row's largest contribute to, against 64 bits and relative to the terms themselves."""
    m, n, k = 300, 264, 136
    rows = (0, 31, 32, 130, 255, 256, 299) if operand == "activations" else (0, 63, 64, 127, 128, 200, 263)
    if form == "all":
        rows = rows[:2]
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    a[:, 0], w[:, 0] = 0.0, 0.0
    if operand == "activations":
        a[list(rows)], w = _tail(a[list(rows)], w, form, low)
    else:
        w[list(rows)], a = _tail(w[list(rows)], a, form, low)
    stream = torch.cuda.current_stream().cuda_stream
    lin = _layer(monkeypatch, "1", m, n, k, w)
    c = torch.empty((m, n), device=cuda_device)
    for _ in range(2):
        lin.run(a, w, c, stream=stream)
    lin.check(stream=stream)
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # each operand to 2^-22, the product of the low parts 2^-22, and per 8 columns three additions that cut at 2^-23 of a partial sum
    bound = (3 * 2.0 ** -22 + (k / 8 * 3 + 8) * 2.0 ** -23) * size
    if form == "few":
        # five terms in five k-steps (and as many rounded to fp32 where they are added one by one)
        part = (list(rows), slice(None)) if operand == "activations" else (slice(None), list(rows))
        bound[part] = (3 * 2.0 ** -22 + (5 * 3 + 5) * 2.0 ** -23) * size[part]
    assert bool(((c.double() - want).abs() <= bound).all())


def test_small_elements_of_both_operands_meet(cuda_device, monkeypatch):
    """A row and a column whose largest elements meet zeros, and whose small ones meet each other, once where both are small."""
    m, n, k = 300, 264, 136
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    a[:, :2], w[:, :2] = 0.0, 0.0
    a[40], w[70] = 0.0, 0.0
    a[40, 0], w[70, 1] = 1.0, 1.0
    a[40, 5], w[70, 5] = 1.7 * 2.0 ** -30, 1.3 * 2.0 ** -31
    a[40, 100], a[40, 130] = 1.1 * 2.0 ** -33, -1.9 * 2.0 ** -29
    w[70, 130] = 1.4 * 2.0 ** -32
    stream = torch.cuda.current_stream().cuda_stream
    lin = _layer(monkeypatch, "1", m, n, k, w)
    tf32, c = torch.empty((m, n), device=cuda_device), torch.empty((m, n), device=cuda_device)
    lin.run(a, w, c, alpha=0.5, stream=stream)
    lin.check(stream=stream)
    assert lin.last_launches == 4
    _layer(monkeypatch, "0", m, n, k, w).run(a, w, tf32, alpha=0.5, stream=stream)
    want, size = 0.5 * (a.double() @ w.double().T), 0.5 * (a.double().abs() @ w.double().abs().T)
    # per term: each operand to 2^-22, the low parts' product 2^-22, rounding of the product and of each sum 2^-23
    assert bool(((c.double() - want).abs()[40, :] <= (3 * 2.0 ** -22 + (3 * 3 + 4) * 2.0 ** -23) * size[40, :]).all())
    assert bool(((c.double() - want).abs()[:, 70] <= (3 * 2.0 ** -22 + (3 * 3 + 4) * 2.0 ** -23) * size[:, 70]).all())
    assert float(want[40, 70]) != 0.0 and not torch.equal(c, tf32)


@pytest.mark.parametrize("operand", ["activations", "weights"])
@pytest.mark.parametrize("rows,per_row,value,planes", [(1, 1, 1e-10, True), (1, 8, 1e-17, True), (16, 1, 1e-12, True), (17, 1, 1e-12, False), (1, 9, 1e-10, False)])
def test_a_few_tiny_elements_stay_on_the_planes(cuda_device, monkeypatch, operand, rows, per_row, value, planes):
    """Beside elements of size one; more rows or elements than the lists take are the TF32 form bit by bit."""
    m, n, k = 300, 520, 328
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    for x in (a, w):
        x.copy_(torch.where(x.abs() < 1e-3, torch.full_like(x, 1e-3), x))
    x = a if operand == "activations" else w
    for r in range(rows):
        x[m - 1 - 17 * r, 40 * r % (k - per_row):][:per_row] = value
    stream = torch.cuda.current_stream().cuda_stream
    tf32, c = torch.empty((m, n), device=cuda_device), torch.empty((m, n), device=cuda_device)
    _layer(monkeypatch, "0", m, n, k, w).run(a, w, tf32, stream=stream)
    lin = _layer(monkeypatch, "1", m, n, k, w)
    lin.run(a, w, c, stream=stream)
    lin.check(stream=stream)
    assert torch.equal(c, tf32) is not planes
    size = a.double().abs() @ w.double().abs().T
    assert bool(((c.double() - a.double() @ w.double().T).abs() <= (3 * 2.0 ** -22 + (k / 8 * 3 + 12) * 2.0 ** -23) * size).all())


def test_scratch_of_a_run_is_that_of_the_tf32_form(cuda_device, monkeypatch):
    m, n, k = 1100, 520, 328
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    stream = torch.cuda.current_stream().cuda_stream
    c, grown = torch.empty((m, n), device=cuda_device), []
    for planes in "01":
        lin = _layer(monkeypatch, planes, m, n, k, w)
        before = lin.workspace_bytes
        lin.run(a, w, c, stream=stream)
        lin.check(stream=stream)
        grown.append(lin.workspace_bytes - before)
    assert grown[1] <= grown[0] + 16


def test_pre_packing_a_new_primitive_allocates_once(cuda_device, monkeypatch):
    m, n, k = 300, 520, 328
    a, w = _draw(cuda_device, m, k), _draw(cuda_device, n, k)
    stream = torch.cuda.current_stream().cuda_stream
    c = torch.empty((m, n), device=cuda_device)
    monkeypatch.setenv("KUDNN_B200_TC_PLANES", "1")
    lin = kb.Linear(kb.make_desc(m, n, k, kb.F32))
    lin.force_kernel(kb.KERNEL_TC)
    try:
        kb.debug_fail_allocation(2)  # the status block, both kinds of planes: a third would fail, and the fp16 planes be left out
        lin.prepack(w, stream=stream)
    finally:
        kb.debug_fail_allocation(-1)
    lin.run(a, w, c, stream=stream)
    lin.check(stream=stream)
    assert lin.last_launches == 4


@pytest.mark.parametrize("n", [2564, 2308])
@pytest.mark.parametrize("marks", [False, True])
def test_several_tiles_per_pair(cuda_device, monkeypatch, n, marks):
    """17 x 11 tiles: two waves on 74 pairs and a third of whole tiles; 17 x 10: the last wave of halves.  Two raster groups, two calls one
    after the other on other inputs, chosen by size."""
    monkeypatch.delenv("KUDNN_B200_TC_PLANES", raising=False)
    m, k = 4100, 264
    w, side = _draw(cuda_device, n, k), _draw(cuda_device, n)
    xs = [_draw(cuda_device, m, k), _draw(cuda_device, m, k + 1)[:, :k].contiguous()]
    for x in xs + [w]:
        x.copy_(torch.where(x.abs() < 1e-3, torch.full_like(x, 1e-3), x))
    if marks:
        xs[0][4099, 77], xs[0][130, 3], w[n - 1, 263] = 1e-11, -2e-10, 3e-9
    stream = torch.cuda.current_stream().cuda_stream
    lin = kb.Linear(kb.make_desc(m, n, k, kb.F32, has_bias=True))
    lin.prepack(w, stream=stream)
    cs = [torch.full((m, n), 7.0, device=cuda_device) for _ in xs]
    for x, c in zip(xs, cs):
        lin.run(x, w, c, side, stream=stream)
    lin.check(stream=stream)
    assert lin.last_launches == 4
    for x, c in zip(xs, cs):
        want = x.double() @ w.double().T + side.double()
        error = c.double() - want
        # every 256 x 128 piece by itself: the operands to 2^-23, and 17 steps of 16 columns, each cut at 2^-23 of the sum so far
        for r in range(0, m, 256):
            for j in range(0, n, 128):
                part = (slice(r, r + 256), slice(j, j + 128))
                assert float(error[part].norm()) <= (k / 16 + 8) * 2.0 ** -23 * float(want[part].norm())


@pytest.mark.parametrize("n,desc", [(1030, {}), (1032, dict(res_op=kb.RES_IDENTICAL)), (1032, dict(act=kb.ACT_TANH)), (1032, dict(c_strides=(1, 1100))),
                                    (1032, dict(has_bias=True, bias_strides=(1, 0))), (1032, dict(a_strides=(1, 1100))), (1032, dict(a_strides=(330, 1)))])
def test_planes_are_not_packed_where_no_run_takes_them(cuda_device, monkeypatch, n, desc):
    m, k = 1100, 328
    w = _draw(cuda_device, n, k)
    held = [_layer(monkeypatch, planes, m, n, k, w, **desc).workspace_bytes for planes in "01"]
    assert held[0] == held[1]


@pytest.mark.parametrize("m,n,k,planes", [(64, 5120, 8192, False), (64, 5120, 4096, True), (64, 6144, 8192, True), (300, 2560, 8192, False),
                                          (256, 5120, 8192, True), (385, 2560, 8192, True)])
def test_few_tiles_that_are_half_empty_stay_on_the_tf32_form_where_k_is_long(cuda_device, monkeypatch, m, n, k, planes):
    monkeypatch.delenv("KUDNN_B200_TC_PLANES", raising=False)
    a, w = _draw(cuda_device, m, k).clamp(1e-3, 4.0), _draw(cuda_device, n, k).clamp(-4.0, -1e-3)
    lin = kb.Linear(kb.make_desc(m, n, k, kb.F32))
    stream = torch.cuda.current_stream().cuda_stream
    lin.prepack(w, stream=stream)
    c = torch.empty((m, n), device=cuda_device)
    lin.run(a, w, c, stream=stream)
    lin.check(stream=stream)
    assert lin.last_launches == (4 if planes else 2)
    want = a.double() @ w.double().T
    # all terms have one sign: 3 k / 8 additions at most, each cut at 2^-23 of the sum
    assert bool(((c.double() - want).abs() <= (3 * 2.0 ** -22 + (k / 8 * 3 + 4) * 2.0 ** -23) * want.abs()).all())
