"""The launch shapes that depend on the problem's size: tile widths and K cuts of the tensor-core kernel with the tile finished
from shared memory, the general kernel for few tiles, row packing, and the cuts of the streaming kernels.  Sizes sit at the
edges: one row or column over a tile, rows that start anywhere, K shorter than a block, the last group of weight rows
incomplete."""
import numpy as np
import pytest
import torch

import kudnn_b200 as kb
from oracle import ko
from tests import helpers

pytestmark = pytest.mark.gpu


def _run(cuda_device, kernel, **case):
    case = dict(dict(x_dist="normal", w_std=0.05, seed=17), **case)
    prepack = case.pop("prepack", False)
    desc, arrays, c = helpers.build_case(case)
    ref_c, ref_o = helpers.run_oracle(desc, arrays, c, acc=ko.ACC_F64)
    got_c, got_o, used = helpers.run_gpu(desc, arrays, c, cuda_device, prepack=prepack)
    assert used == kernel
    if c["want_c"]:
        helpers.compare(got_c, ref_c, desc.c_dtype)
    if desc.res_op != kb.RES_NONE:
        helpers.compare(got_o, ref_o, desc.out_dtype)


@pytest.mark.parametrize("dtype", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("m,n,k", [(17, 2561, 1030), (129, 1040, 2050), (333, 3001, 264), (257, 48, 4104), (24, 19208, 72)])
@pytest.mark.parametrize("act,res_op", [(kb.ACT_GELU_ERF, kb.RES_NONE), (kb.ACT_NONE, kb.RES_IDENTICAL)])
@pytest.mark.parametrize("layout", ["BA", "AB"])
def test_tile_widths_and_cuts(cuda_device, dtype, m, n, k, act, res_op, layout):
    _run(cuda_device, kb.KERNEL_TC, m=m, n=n, k=k, dtype=dtype, bias="row", act=act, res_op=res_op, b_layout=layout,
         prepack=n % 2 == 0)


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("splits", ["1", "2", "4", "8"])
@pytest.mark.parametrize("n", [130, 136])
@pytest.mark.parametrize("bias", ["row", "full"])
def test_every_cut_of_k(cuda_device, monkeypatch, capfd, dtype, splits, n, bias):
    monkeypatch.setenv("KUDNN_B200_TC_SPLITS", splits)
    monkeypatch.setenv("KUDNN_B200_DEBUG", "1")
    _run(cuda_device, kb.KERNEL_TC, m=133, n=n, k=1500, dtype=dtype, bias=bias, act=kb.ACT_SWISH, res_op=kb.RES_NONE)
    assert "k splits %s," % splits in capfd.readouterr().err


@pytest.mark.parametrize("dtype", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("m,n,k", [(33, 65, 1), (31, 33, 15), (113, 198, 246), (64, 1600, 65), (18, 17, 300)])
@pytest.mark.parametrize("layout", ["BA", "AB"])
def test_few_tiles_on_the_general_kernel(cuda_device, dtype, m, n, k, layout):
    _run(cuda_device, kb.KERNEL_SIMT, m=m, n=n, k=k, dtype=dtype, bias="row", act=kb.ACT_SWISH, res_op=kb.RES_IDENTICAL, b_layout=layout)


@pytest.mark.parametrize("m,n,k,kernel", [(24, 64, 8192, kb.KERNEL_TC), (17, 256, 2000, kb.KERNEL_TC), (128, 256, 256, kb.KERNEL_TC),
                                          (128, 512, 200, kb.KERNEL_SIMT), (76, 1562, 73, kb.KERNEL_SIMT)])
def test_small_fp32_goes_by_the_length_of_k(cuda_device, m, n, k, kernel):
    _run(cuda_device, kernel, m=m, n=n, k=k, dtype="f32", bias="row", act=kb.ACT_RELU, act_alpha=0.0, res_op=kb.RES_NONE)


@pytest.mark.parametrize("m,n,k", [(1, 1000, 8200), (1, 70, 16384), (3, 520, 4104), (8, 1003, 6152), (9, 2000, 5896), (16, 24, 8192),
                                   (2, 9001, 32), (5, 7, 40), (12, 200, 72), (1, 20000, 264), (1, 3, 32), (8, 28003, 1040)])
@pytest.mark.parametrize("prepack", [False, True])
def test_streaming_cuts(cuda_device, m, n, k, prepack):
    kernel = kb.KERNEL_GEMV_FMA if m == 1 else kb.KERNEL_GEMV_MMA
    _run(cuda_device, kernel, m=m, n=n, k=k, dtype="bf16", bias="row", act=kb.ACT_SWISH, res_op=kb.RES_NONE, prepack=prepack)


@pytest.mark.parametrize("m,n,k", [(1, 5000, 516), (2, 9001, 36), (4, 209, 1156), (3, 70, 8196), (1, 300, 20484)])
@pytest.mark.parametrize("prepack", [False, True])
def test_streaming_cuts_fp32(cuda_device, m, n, k, prepack):
    _run(cuda_device, kb.KERNEL_GEMV_FMA, m=m, n=n, k=k, dtype="f32", bias="row", act=kb.ACT_SWISH, res_op=kb.RES_IDENTICAL, prepack=prepack)


@pytest.mark.parametrize("wcode", [kb.S8, kb.U8])
@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(15, 8208), (1003, 1040), (2464, 5264), (9001, 48)])
def test_streaming_8_bit_weights(cuda_device, wcode, m, n, k):
    rng = np.random.default_rng(5)
    x = ko.to_storage(rng.standard_normal((1, m, k), dtype=np.float32), kb.F16)
    lo, hi = (-128, 128) if wcode == kb.S8 else (0, 256)
    arrays = {"a": x, "b": rng.integers(lo, hi, (1, n, k)).astype(ko.np_dtype(wcode))}
    desc = kb.make_desc(m, n, k, kb.F16, b_dtype=wcode)
    c = helpers.case_defaults(dict(m=m, n=n, k=k, res_op=kb.RES_NONE))
    ref, _ = helpers.run_oracle(desc, arrays, c, acc=ko.ACC_F64)
    for prepack in (False, True):
        got, _, used = helpers.run_gpu(desc, arrays, c, cuda_device, prepack=prepack)
        assert used == (kb.KERNEL_GEMV_FMA if m == 1 else kb.KERNEL_GEMV_MMA)
        helpers.compare(got, ref, desc.c_dtype)


# rows, width, whether the CTA pairs are asked for, what the plan must say (None: another kernel)
_CHAINS = [(1, 512, False, None), (4, 512, False, None), (12, 512, False, None), (33, 72, False, None), (40, 512, False, "128 x"),
           (300, 512, False, "128 x"), (300, 1030, False, "128 x"), (300, 512, True, "256 (CTA pair)"), (300, 1030, True, "256 (CTA pair)")]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("owned", [False, True])
@pytest.mark.parametrize("m,width,pairs,plan", _CHAINS)
def test_chained_calls_read_each_others_results(cuda_device, monkeypatch, capfd, dtype, owned, m, width, pairs, plan):
    """Layers whose input is the previous layer's output, across the kernels that may start before it has ended: packed and split
    activations, and weights in a packed copy (owned: stored [k, n]; fp32 always), the first of which are loaded early."""
    if pairs and width == 1030:
        width = 1032  # rows that are no vectors are left to single CTAs at this size
    if pairs:
        monkeypatch.setenv("KUDNN_B200_TC_PAIR", "1")
    monkeypatch.setenv("KUDNN_B200_DEBUG", "1")
    rng = np.random.default_rng(9)
    stream = torch.cuda.current_stream().cuda_stream
    code = kb.BF16 if dtype == torch.bfloat16 else kb.F32
    ws = [torch.from_numpy(rng.standard_normal((width, width), dtype=np.float32) / width ** 0.5).to(cuda_device, dtype) for _ in range(6)]
    lins = [kb.Linear(kb.make_desc(m, width, width, code, b_strides=(width, 1) if owned else (1, width))) for _ in ws]
    for lin, w in zip(lins, ws):
        lin.prepack(w, stream=stream)
    x = torch.from_numpy(rng.standard_normal((m, width), dtype=np.float32)).to(cuda_device, dtype)
    want = x.double()
    for w in ws:
        want = (want @ (w.double() if owned else w.double().T)).to(dtype).double()
    # six roundings to 8 significant bits, each at most 2^-8 of a value of order one, and what they grow to; fp32: sums of up to
    # 1032 products whose errors of 2^-22 (three TF32 products) add as a random walk, in six layers
    atol, rtol = (6 * 2.0 ** -8 * 4, 2.0 ** -6) if dtype == torch.bfloat16 else (6 * 2.0 ** -22 * 1032 ** 0.5 * 4, 2.0 ** -16)
    for _ in range(20):
        bufs = [torch.full((m, width), float("nan"), device=cuda_device, dtype=dtype) for _ in ws]
        src = x
        for lin, w, dst in zip(lins, ws, bufs):
            lin.run(src, w, dst, stream=stream)
            src = dst
        assert torch.allclose(src.double(), want, atol=atol, rtol=rtol)
    said = capfd.readouterr().err
    assert plan is None or plan in said
    for lin in lins:
        lin.close()


@pytest.mark.parametrize("m", [40, 300])
def test_chained_integer_products(cuda_device, m):
    """Integer tiles of up to 128 columns leave room for two CTAs on an SM: those of consecutive launches share its tensor memory."""
    rng = np.random.default_rng(10)
    stream = torch.cuda.current_stream().cuda_stream
    n, k = 3000, 1040
    a = torch.from_numpy(rng.integers(-128, 128, (4, m, k)).astype(np.int8)).to(cuda_device)
    b = torch.from_numpy(rng.integers(-128, 128, (k, n)).astype(np.int8)).to(cuda_device)
    want = (a.double() @ b.double()).to(torch.int32)
    desc = kb.make_desc(m, n, k, kb.S8, c_dtype=kb.S32, b_strides=(n, 1))
    lin = kb.Linear(desc)
    lin.prepack(b, stream=stream)
    got = torch.zeros((60, m, n), dtype=torch.int32, device=cuda_device)
    for i in range(60):
        lin.run(a[i % 4], b, got[i], stream=stream)
    lin.check(stream=stream)
    assert lin.last_kernel == kb.KERNEL_TC
    assert all(torch.equal(got[i], want[i % 4]) for i in range(60))


@pytest.mark.parametrize("kernel,m", [(kb.KERNEL_GEMV_FMA, 1), (kb.KERNEL_GEMV_FMA, 3), (kb.KERNEL_TC, 40)])
def test_weights_in_place_are_read_after_the_kernel_that_writes_them(cuda_device, kernel, m):
    """Rows used where the caller keeps them are not requested early, whatever other copy a primitive has."""
    rng = np.random.default_rng(12)
    stream = torch.cuda.current_stream().cuda_stream
    n, k = 1024, 512
    parts = torch.from_numpy(rng.standard_normal((20, n, 64), dtype=np.float32)).to(cuda_device, torch.bfloat16)
    mix = torch.from_numpy(rng.standard_normal((k, 64), dtype=np.float32) / 8).to(cuda_device, torch.bfloat16)
    x = torch.from_numpy(rng.standard_normal((m, k), dtype=np.float32)).to(cuda_device, torch.bfloat16)
    w = torch.zeros((n, k), device=cuda_device, dtype=torch.bfloat16)
    y = torch.zeros((20, m, n), device=cuda_device, dtype=torch.bfloat16)
    writer, reader = kb.Linear(kb.make_desc(n, k, 64, kb.BF16)), kb.Linear(kb.make_desc(m, n, k, kb.BF16))
    reader.force_kernel(kernel)
    reader.prepack(w, stream=stream)
    for i in range(20):
        writer.run(parts[i], mix, w, stream=stream)
        reader.run(x, w, y[i], stream=stream)
    for i in range(20):
        want = x.float() @ (parts[i].float() @ mix.float().T).to(torch.bfloat16).float().T
        # one rounding of the result, and weights that round the other way (2^-8 of each of the 512 terms, added as a random walk)
        assert torch.allclose(y[i].float(), want, atol=2.0 ** -8 * 512 ** 0.5, rtol=2.0 ** -8)


@pytest.mark.parametrize("dtype,ctype", [("bf16", "bf16"), ("f16", "f16"), ("f32", "f32"), ("bf16", "f32")])
@pytest.mark.parametrize("n", [136, 132, 131, 129])
@pytest.mark.parametrize("m,pairs", [(133, False), (20, False), (300, True)])
@pytest.mark.parametrize("beta,both", [(0.5, False), (0.5, True), (0.0, True)])
def test_rows_of_vectors_with_beta_and_a_cut_last_column(cuda_device, monkeypatch, dtype, ctype, n, m, pairs, beta, both):
    """c is read and written, rows start on 16 bytes and end inside a vector: nothing beyond column n is touched."""
    if pairs:
        monkeypatch.setenv("KUDNN_B200_TC_PAIR", "1")
    td = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
    code = {"f32": kb.F32, "f16": kb.F16, "bf16": kb.BF16}
    k, gen = 520, torch.Generator(device=cuda_device)
    gen.manual_seed(21)

    def draw(*shape, dt=td[dtype], std=1.0):
        return (torch.randn(shape, generator=gen, device=cuda_device) * std).to(dt)

    vec = 16 // td[ctype].itemsize
    pitch = (n + vec - 1) // vec * vec
    a, w, bias = draw(m, k), draw(n, k, std=0.05), draw(n, dt=td[ctype])
    c, res, out = (draw(m, pitch, dt=td[ctype]) for _ in range(3))
    c0, out0 = c.clone(), out.clone()
    desc = kb.make_desc(m, n, k, code[dtype], c_dtype=code[ctype], has_bias=True, bias_dtype=code[ctype], act=kb.ACT_RELU, act_alpha=0.0,
                        res_op=kb.RES_IDENTICAL if both else kb.RES_NONE, res_dtype=code[ctype], out_dtype=code[ctype],
                        c_strides=(pitch, 1), res_strides=(pitch, 1), out_strides=(pitch, 1))
    lin = kb.Linear(desc)
    lin.force_kernel(kb.KERNEL_TC)
    lin.run(a, w, c, bias, res if both else None, out if both else None, beta=beta, stream=torch.cuda.current_stream().cuda_stream)
    lin.check(stream=torch.cuda.current_stream().cuda_stream)
    want = (a.double() @ w.double().T + beta * c0[:, :n].double() + bias.double()).relu()
    # 16-bit results: a rounding after the bias and one after the second operator.  fp32: up to 195 additions to an accumulator of
    # up to 6, each cut at 2^-23 of it, as a random walk (10^-5)
    eps = {"bf16": 2.0 ** -8, "f16": 2.0 ** -11, "f32": 2.0 ** -16}[ctype]
    assert torch.allclose(c[:, :n].double(), want, rtol=3 * eps, atol=4 * eps)
    assert torch.equal(c[:, n:], c0[:, n:])
    if both:
        assert torch.allclose(out[:, :n].double(), want + res[:, :n].double(), rtol=3 * eps, atol=8 * eps)
        assert torch.equal(out[:, n:], out0[:, n:])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cut,m,n,k", [("1", 129, 512, 64), ("1", 300, 1288, 200), ("1", 1027, 776, 1096), ("2", 257, 520, 8), ("2", 513, 1032, 328),
                                       ("3", 300, 264, 456), ("3", 2000, 1160, 136), (None, 2500, 9992, 264)])
@pytest.mark.parametrize("act,res_op,bias,alpha", [(kb.ACT_NONE, kb.RES_NONE, None, 1.0), (kb.ACT_RELU, kb.RES_IDENTICAL, "row", 1.0),
                                                   (kb.ACT_SWISH, kb.RES_NONE, "row", 1.0), (kb.ACT_GELU_TANH, kb.RES_EXT, "one", 1.0),
                                                   (kb.ACT_NONE, kb.RES_ELTWISE_MUL, "row", 0.75), (kb.ACT_SWISH, kb.RES_IDENTICAL, None, 0.75)])
def test_wide_tiles_equal_the_narrow_ones(cuda_device, monkeypatch, capfd, dtype, cut, m, n, k, act, res_op, bias, alpha):
    """Tiles of 512 columns, whole (1), in halves (2), in quarters (3) and as planned, against the tiles of 256: the same products
    in the same order.  Rows and columns past the tiles' edges, a tile whose second half is empty, outputs and residuals with a
    pitch, one call after the other on the same stream."""
    stream = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(31)

    def draw(*shape, std=1.0):
        return (torch.randn(shape, generator=gen, device=cuda_device) * std).to(dtype)

    code = kb.BF16 if dtype == torch.bfloat16 else kb.F16
    pitch, res_pitch = n + 8, n + 24
    second = res_op != kb.RES_NONE
    owned = k % 16 == 8  # weights stored [k, n]: packed into a copy whose first rows are loaded early
    xs, w, res = [draw(m, k), draw(m, k)], draw(*((k, n) if owned else (n, k)), std=0.05), draw(m, res_pitch)
    side = draw(n) if bias == "row" else draw(1) if bias == "one" else None
    desc = kb.make_desc(m, n, k, code, b_strides=(n, 1) if owned else None, has_bias=bias is not None,
                        bias_strides=(0, 0) if bias == "one" else None, act=act, act_alpha=0.25,
                        res_op=res_op, c_strides=(pitch, 1), res_strides=(res_pitch, 1), out_strides=(pitch, 1))
    monkeypatch.setenv("KUDNN_B200_DEBUG", "1")
    got = []
    for wide in ("0", cut):
        for name, value in (("KUDNN_B200_TC_WIDE", wide), ("KUDNN_B200_TC_PAIR", "1" if wide == "0" else None)):
            monkeypatch.delenv(name, raising=False) if value is None else monkeypatch.setenv(name, value)
        lin = kb.Linear(desc)
        lin.force_kernel(kb.KERNEL_TC)
        lin.prepack(w, stream=stream)
        ys = [torch.full((m, pitch), 7.0, device=cuda_device, dtype=dtype) for _ in xs]
        for x, y in zip(xs, ys):
            lin.run(x, w, None if second else y, side, res if second else None, y if second else None, alpha=alpha, gamma=0.5, stream=stream)
        lin.check(stream=stream)
        said = capfd.readouterr().err
        assert ("256 (CTA pair) x 512" in said) == (wide != "0")
        got.append(ys)
        lin.close()
    for a, b in zip(*got):
        assert bool((b[:, n:] == 7.0).all())
        if alpha == 1.0:
            assert torch.equal(a, b)
        else:
            # alpha * acc + bias is rounded once here and twice there: one unit of the 16-bit value, carried through the chain
            eps = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
            assert torch.allclose(a.float(), b.float(), rtol=2 * eps, atol=2 * eps)


@pytest.mark.parametrize("cut,m,n,k", [("1", 129, 512, 128), ("1", 1027, 776, 1096), ("2", 257, 516, 16), ("2", 513, 1032, 640), ("3", 300, 264, 912),
                                       ("3", 2000, 1160, 272), (None, 4100, 9004, 520), (None, 4100, 9001, 520)])
@pytest.mark.parametrize("signs", [(kb.S8, kb.S8), (kb.U8, kb.S8)])
@pytest.mark.parametrize("bias", [False, True])
def test_wide_tiles_of_integer_products(cuda_device, monkeypatch, capfd, cut, m, n, k, signs, bias):
    """8-bit integers on tiles of 512 columns: exact, also where the sum with the bias leaves the 32-bit range."""
    stream = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(41)

    def draw(code, *shape):
        lo, hi, dt = (-128, 128, torch.int8) if code == kb.S8 else (0, 256, torch.uint8)
        return torch.randint(lo, hi, shape, generator=gen, device=cuda_device, dtype=torch.int32).to(dt)

    if cut is not None:
        monkeypatch.setenv("KUDNN_B200_TC_WIDE", cut)
    monkeypatch.setenv("KUDNN_B200_DEBUG", "1")
    a, w = draw(signs[0], m, k), draw(signs[1], n, k)
    side = torch.randint(-2 ** 31, 2 ** 31 - 1, (n,), generator=gen, device=cuda_device, dtype=torch.int64).to(torch.int32) if bias else None
    pitch = (n + 3) // 4 * 4 + 4
    lin = kb.Linear(kb.make_desc(m, n, k, signs[0], b_dtype=signs[1], c_dtype=kb.S32, has_bias=bias, bias_dtype=kb.S32, c_strides=(pitch, 1)))
    lin.force_kernel(kb.KERNEL_TC)
    lin.prepack(w, stream=stream)
    c = torch.full((m, pitch), 7, device=cuda_device, dtype=torch.int32)
    for _ in range(2):
        lin.run(a, w, c, side, stream=stream)
    lin.check(stream=stream)
    want = a.double() @ w.double().T + (side.double() if bias else 0.0)
    assert torch.equal(c[:, :n], want.clamp(-2.0 ** 31, 2.0 ** 31 - 1).to(torch.int64).to(torch.int32))
    assert bool((c[:, n:] == 7).all())
    assert ("256 (CTA pair) x 512" in capfd.readouterr().err) == (n % 4 == 0)  # rows that end inside 16 bytes are left to narrow tiles


@pytest.mark.parametrize("kind", [kb.BF16, kb.F16])
@pytest.mark.parametrize("cut", ["1", "2", "3"])
@pytest.mark.parametrize("wide_bias", [False, True])
def test_wide_tiles_round_alpha_times_the_product(cuda_device, monkeypatch, kind, cut, wide_bias):
    """alpha * acc is rounded to fp32 (to fp16 in the fp16 chain) ahead of the bias, in tiles of any width: the same bits, so that
    the rows of a call may be cut anywhere."""
    m, n, k = 1200, 2056, 264
    dtype = torch.bfloat16 if kind == kb.BF16 else torch.float16
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(43)
    a, w, side = (torch.randn(s, generator=gen, device=cuda_device).to(dtype) for s in ((m, k), (n, k), (n,)))
    stream = torch.cuda.current_stream().cuda_stream
    got = []
    for wide in ("0", cut):
        monkeypatch.setenv("KUDNN_B200_TC_WIDE", wide)
        lin = kb.Linear(kb.make_desc(m, n, k, kind, has_bias=True, bias_dtype=kb.F32 if wide_bias else None, act=kb.ACT_RELU, act_alpha=0.25))
        lin.force_kernel(kb.KERNEL_TC)
        lin.prepack(w, stream=stream)
        c = torch.empty((m, n), device=cuda_device, dtype=dtype)
        lin.run(a, w, c, side.float() if wide_bias else side, alpha=0.3, stream=stream)
        lin.check(stream=stream)
        got.append(c)
    assert torch.equal(*got)


@pytest.mark.parametrize("kind", [kb.BF16, kb.F16])
@pytest.mark.parametrize("alpha,n,pitch", [(1.0, 2056, 2056), (0.3, 2056, 2056), (1.0, 2052, 2056), (0.3, 2052, 2056), (1.0, 2051, 2051), (1.0, 2052, 2052)])
def test_gelu_is_the_same_in_every_epilogue(cuda_device, monkeypatch, kind, alpha, n, pitch):
    """Finished from tensor memory, from shared memory or on wide tiles, in whole vectors, cut ones or value by value: the same bits."""
    m, k = 1200, 264
    dtype = torch.bfloat16 if kind == kb.BF16 else torch.float16
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(47)
    a, w = (torch.randn(s, generator=gen, device=cuda_device).to(dtype) for s in ((m, k), (n, k)))
    a *= 0.2  # results of a few units, where the forms of the function differ most
    stream = torch.cuda.current_stream().cuda_stream
    got = []
    for pair, wide in (("1", "0"), ("0", "0"), (None, "1")):
        for name, value in (("KUDNN_B200_TC_PAIR", pair), ("KUDNN_B200_TC_WIDE", wide), ("KUDNN_B200_TC_SPLITS", "1")):
            monkeypatch.delenv(name, raising=False) if value is None else monkeypatch.setenv(name, value)
        lin = kb.Linear(kb.make_desc(m, n, k, kind, act=kb.ACT_GELU_TANH, c_strides=(pitch, 1)))
        lin.force_kernel(kb.KERNEL_TC)
        lin.prepack(w, stream=stream)
        c = torch.zeros((m, pitch), device=cuda_device, dtype=dtype)
        lin.run(a, w, c, alpha=alpha, stream=stream)
        lin.check(stream=stream)
        got.append(c)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
