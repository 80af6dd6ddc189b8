"""Packed FP4 weights on the fp16 form: row conversion, dense and grouped products at the edges of tiles, and which weights take it."""
import pytest
import torch

from fllm_b200.ops.fp4 import Fp4ExpertStack, Fp4Weight, dequantize_fp4, fp16_form


@pytest.fixture(scope="module")
def ops():
    from fllm_b200.ops import get_ops
    return get_ops(torch.device("cuda:0"))


def _rand(shape, seed, std=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std).to(torch.bfloat16)


def _rel(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


def test_which_weights_are_exact_in_fp16():
    codes = torch.full((2, 32), 0x77, dtype=torch.uint8)
    scales = torch.full((2, 2), 120, dtype=torch.uint8)
    assert fp16_form(codes, scales, 1) and fp16_form(codes, scales, 0)
    for s, ok in ((104, True), (103, False), (140, True), (141, False), (0, True), (255, False)):
        scales[1, 1] = s
        assert fp16_form(codes, scales, 1) == ok
    codes[1, 16:] = 0x88                       # zeros (of either sign) need no scale, unless it is not a number
    for s, ok in ((1, True), (103, True)):
        scales[1, 1] = s
        assert fp16_form(codes, scales, 1) == ok


def test_zeros_under_a_scale_that_fp16_does_not_hold():
    """Scales from 2^16 on (byte 143) are infinite in fp16, and zero times that is not a number."""
    codes = torch.full((2, 32), 0x77, dtype=torch.uint8)
    codes[1, 16:] = 0x80
    scales = torch.full((2, 2), 120, dtype=torch.uint8)
    for s, ok in ((141, True), (142, True), (143, False), (200, False), (255, False)):
        scales[1, 1] = s
        assert fp16_form(codes, scales, 1) == ok


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [142, 143, 200])
def test_blocks_of_zeros_under_large_scales(ops, scale):
    q = Fp4Weight.from_dense(_rand((256, 512), 2, 0.05).cuda(), "mxfp4")
    q.codes[7, 32:48], q.scales[7, 2] = 0, scale
    q = Fp4Weight(q.codes, q.scales, 1)
    x = _rand((24, 512), 1).cuda()
    assert _rel(ops.linear(x, q), x.double() @ dequantize_fp4(q.codes, q.scales, 1).double().t()) < 2.5e-3
    stack = Fp4ExpertStack(q.codes[None], q.scales[None], 1)
    assert stack.f16 == q.f16 == (scale < 143)


def test_one_factor_for_an_activation_needs_room_below():
    from fllm_b200.models.moe import _oai_scale
    assert _oai_scale(1.702, 7.0) == 1024.0 and _oai_scale(1.702, 0.5) == 4096.0
    for limit in (8.0, 100.0, 240.0, 1e6, 0.0):
        assert _oai_scale(1.702, limit) == 0.0
    assert _oai_scale(1e-3, 7.0) == 0.0


def _experts(ops, counts, k, act, limit=7.0, size=1.0, weigh=False, alpha=1.702):
    """moe_ffn over MXFP4 experts, expert e chosen by counts[e] (token, place) pairs, and the same in 64 bits. The first values of a row are
    its router logits (times ``size``)."""
    from types import SimpleNamespace
    from fllm_b200.config import ModelConfig, MoeSpec
    from fllm_b200.models.moe import moe_ffn
    from fllm_b200.models.weights import LayerWeights
    E, H, I, T = len(counts), 256, 192, sum(counts) // k
    cfg = ModelConfig(hidden_size=H, num_experts=E, experts_per_token=k, moe_intermediate_size=I, act=act, swiglu_limit=limit, swiglu_alpha=alpha)
    lw = LayerWeights(attn_norm=None, wqkv=None, wo=None, ffn_norm=None)
    lw.moe = MoeSpec(E, k, act=act, weigh_input=weigh)
    lw.router_w = torch.eye(max(E, 8), H, dtype=torch.bfloat16, device="cuda")[:E]
    lw.exp_gate_up, lw.exp_down = Fp4ExpertStack.from_dense(_rand((E, 2 * I, H), 3, 0.01).cuda()), Fp4ExpertStack.from_dense(_rand((E, H, I), 5, 0.05).cuda())
    ids = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)]).view(k, T).t()
    h = _rand((T, H), 7)
    h[:, :E] = 0
    h.scatter_(1, ids, torch.tensor([[4.0, 3.0, 2.5, 2.0][:k]]).expand(T, k).to(torch.bfloat16))
    h = (h * size).cuda()
    w = torch.softmax(torch.tensor([[4.0, 3.0, 2.5, 2.0][:k]]).double() * size, -1)
    got = moe_ffn(SimpleNamespace(cfg=cfg, ops=ops, spec=SimpleNamespace(expert_parallel=False, expert_start=0)), lw, h)
    gu, dn, ref = lw.exp_gate_up.dense().double(), lw.exp_down.dense().double(), torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for j in range(k):
        for e in range(E):
            t = (ids[:, j] == e).nonzero().flatten().cuda()
            x = h[t].double() * (w[0, j].item() if weigh else 1.0)
            u = x @ gu[e].t()
            if act == "swiglu_oai":
                g, u = u[:, 0::2].clamp(max=limit), u[:, 1::2].clamp(-limit, limit)
                u = g * torch.sigmoid(alpha * g) * (u + 1)
            else:
                u = torch.nn.functional.silu(u[:, :I]) * u[:, I:]
            ref[t] += u @ dn[e].t() * (1.0 if weigh else w[0, j].item())
    assert ops.check_status() == 0
    return _rel(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [7.0, 100.0, 240.0])
@pytest.mark.parametrize("size", [1.0, 2.0 ** -10, 2.0 ** -18])
def test_small_activations_of_experts(ops, limit, size):
    """Activations of 2^-5, 2^-15 and 2^-23 under limits that leave them room above. Rounded to bf16 are gate and up, the activation, an
    expert's result and their sum: four roundings of 0.17 % in the mean square."""
    assert _experts(ops, [5, 4, 0, 9], 2, "swiglu_oai", limit, size) < 4 * 1.7e-3


@pytest.mark.gpu
@pytest.mark.parametrize("counts,k", [((0, 1, 96, 97, 106), 1), ((5, 4, 0, 9), 2), ((70, 1, 0, 71), 1), ((1, 0, 0, 0, 0, 0, 0, 0), 1)])
@pytest.mark.parametrize("act,limit", [("swiglu_oai", 7.0), ("swiglu_oai", 100.0), ("swiglu", 7.0)])
@pytest.mark.parametrize("weigh", [False, True])
def test_routed_experts_end_to_end(ops, counts, k, act, limit, weigh):
    """Both ways from gate and up to the rows of the second product, weights on an expert's input or output, experts of 0, 1, 96 and 97 rows
    on the tiles that the mean of them chooses (96 for the first). Roundings to bf16: gate and up, the activation, an expert's result,
    their sum and a weighted input; 0.17 % in the mean square each."""
    from fllm_b200.models.moe import _packed_tile
    assert _packed_tile(sum(counts) / len(counts)) == {5: 96, 4: 64 if k == 1 else 16, 8: 16}[len(counts)]
    assert _experts(ops, counts, k, act, limit, weigh=weigh) < 5 * 1.7e-3


@pytest.mark.gpu
@pytest.mark.parametrize("counts,k,tile", [((65, 97, 106, 0), 1, 96), ((130, 129, 1), 1, 128), ((100, 70, 110), 2, 128), ((1, 0, 299), 1, 128)])
@pytest.mark.parametrize("act,limit", [("swiglu_oai", 7.0), ("swiglu_oai", 100.0), ("swiglu", 7.0)])
@pytest.mark.parametrize("weigh", [False, True])
def test_many_rows_an_expert_end_to_end(ops, counts, k, tile, act, limit, weigh):
    """More than 64 rows an expert in the mean: MXFP4 stacks are expanded to fp16, on tiles of 96 and 128. Roundings as in
    test_routed_experts_end_to_end."""
    from types import SimpleNamespace
    from fllm_b200.models.moe import _mx_tile, _packed_tile
    mean = sum(counts) / len(counts)
    stack = SimpleNamespace(atoms=torch.empty(1))
    assert _mx_tile(SimpleNamespace(exp_gate_up=stack, exp_down=stack), mean) == 0 and _packed_tile(mean) == tile
    assert _experts(ops, counts, k, act, limit, weigh=weigh) < 5 * 1.7e-3


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [7.0, 100.0, 240.0])
@pytest.mark.parametrize("size", [1.0, 2.0 ** -10, 2.0 ** -18])
def test_small_activations_of_many_rows(ops, limit, size):
    """As test_small_activations_of_experts, with more than 64 rows an expert: one factor for all rows of the activation, and rows
    converted again under the limits that leave it too little."""
    assert _experts(ops, [90, 70, 50], 2, "swiglu_oai", limit, size) < 4 * 1.7e-3


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0, 16, 32])
@pytest.mark.parametrize("act", ["swiglu_oai", "swiglu"])
def test_stacks_that_start_on_16_bytes(ops, monkeypatch, at, act):
    """Codes that are a view into a larger buffer: the block-scaled form takes those on 32 bytes, the fp16 form the others. Roundings as in
    test_routed_experts_end_to_end."""
    plain, made = Fp4ExpertStack.from_dense, []

    def moved(w):
        s = plain(w)
        buf = torch.empty(s.codes.numel() + 64, dtype=torch.uint8, device="cuda")
        assert buf.data_ptr() % 32 == 0
        made.append(Fp4ExpertStack(buf[at:at + s.codes.numel()].view(s.codes.shape).copy_(s.codes), s.scales, s.fmt))
        return made[-1]
    monkeypatch.setattr(Fp4ExpertStack, "from_dense", staticmethod(moved))
    assert _experts(ops, [5, 4, 0, 9], 2, act) < 5 * 1.7e-3
    assert len(made) == 2 and all((s.atoms is None) == (at == 16) and s.codes.data_ptr() % 32 == at % 32 for s in made)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [64, 320, 2880, 28672])
def test_rows_keep_every_value(ops, K):
    """fp16 rows times their factor are the bf16 rows again, over the whole exponent range and next to values that are not finite. A value
    below 2^-31 of the row's largest, whose 8 bits reach under the smallest fp16 step of 2^-24, may be off by half of that step."""
    x = _rand((9, K), 1)
    x[0] *= 2.0 ** 100
    x[1] *= 2.0 ** -110
    x[2] = 0
    x[3, 1::2] *= 2.0 ** -20
    x[4, 5], x[5, 6], x[5, 7] = float("nan"), float("inf"), -float("inf")
    x[6] = torch.finfo(torch.bfloat16).max
    xh, f = torch.empty(11, K, dtype=torch.float16, device="cuda"), torch.empty(11, device="cuda")
    token_of = torch.tensor([0, -1, 1, 2, 3, 4, 5, 6, 7, 8, -1], dtype=torch.int32, device="cuda")
    ops.k.moe_rows_f16(x.cuda(), token_of, xh, f)
    back = (xh.double() * f.double()[:, None]).cpu()
    rows = [i for i in range(11) if token_of[i] >= 0]
    xd = x.double()
    finite = xd.isfinite()
    assert torch.equal(back[rows][~finite].nan_to_num(5.0), xd[~finite].nan_to_num(5.0))
    off = torch.where(finite, (back[rows] - xd).abs(), 0)
    top = torch.where(finite, xd.abs(), 0).amax(1, keepdim=True)
    assert (off <= f.double().cpu()[rows][:, None] * 2.0 ** -25).all() and (off[finite & (xd.abs() >= top * 2.0 ** -31)] == 0).all()
    assert (back[[1, 10]] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp4"])
@pytest.mark.parametrize("T,N,K", [(5, 128, 64), (17, 136, 192), (64, 256, 1088), (65, 1000, 320), (96, 264, 3072), (97, 264, 832), (128, 40960, 256), (128, 512, 12288)])
def test_dense_against_64_bits(ops, fmt, T, N, K):
    """One rounding to bf16 (2^-9 of a value at most, 0.17 % in the mean square) is all that a correct product is off."""
    x, q = _rand((T, K), 1).cuda(), Fp4Weight.from_dense(_rand((N, K), 2, 0.05).cuda(), fmt)
    assert q.f16
    x[0] *= 2.0 ** 40
    y = ops.linear(x, q)
    ref = x.double() @ dequantize_fp4(q.codes, q.scales, q.fmt, 1.0).double().t() * q.alpha
    assert _rel(y[:1], ref[:1]) < 2.5e-3 and _rel(y[1:], ref[1:]) < 2.5e-3
    assert ops.check_status() == 0


@pytest.mark.gpu
def test_scales_beyond_fp16_take_the_bf16_form(ops):
    q = Fp4Weight.from_dense(_rand((256, 512), 2, 0.05).cuda(), "mxfp4")
    q = Fp4Weight(q.codes, q.scales - 60, 1)
    assert not q.f16
    x = _rand((24, 512), 1).cuda()
    assert _rel(ops.linear(x, q), x.double() @ dequantize_fp4(q.codes, q.scales, 1).double().t()) < 2.5e-3


@pytest.mark.gpu
@pytest.mark.parametrize("bn", [16, 32, 64, 96, 128])
@pytest.mark.parametrize("n,k", [(32, 64), (304, 192), (5760, 2880)])
@pytest.mark.parametrize("glu", [False, True])
def test_grouped(ops, bn, n, k, glu):
    """Experts with no row, one row, a full tile and one more than that; the clamped activation in the epilogue."""
    counts = [0, 1, bn, bn + 1, 7]
    E = len(counts)
    q = Fp4ExpertStack.from_dense(_rand((E, n, k), 3, 0.05).cuda())
    bias = _rand((E, n), 4, 0.1).cuda()
    tiles = [(e, j) for e, c in enumerate(counts) for j in range(-(-c // bn))]
    rows = len(tiles) * bn
    tile_e = torch.tensor([e for e, _ in tiles] + [0] * 3, dtype=torch.int32, device="cuda")
    tile_r = torch.arange(len(tiles) + 3, dtype=torch.int32, device="cuda") * bn
    real = torch.cat([torch.arange(bn) + j * bn < counts[e] for e, j in tiles]).cuda()
    x = _rand((rows, k), 5).cuda()
    token_of = torch.where(real, torch.arange(rows, device="cuda"), -1).int()
    xh, f = torch.empty(rows, k, dtype=torch.float16, device="cuda"), torch.empty(rows, device="cuda")
    ops.k.moe_rows_f16(x, token_of, xh, f)
    y = torch.empty(rows, n // 2 if glu else n, dtype=torch.float16 if glu else torch.bfloat16, device="cuda")
    num = torch.tensor([len(tiles), rows], dtype=torch.int32, device="cuda")
    ops.k.moe_grouped_linear_w4_f16(xh, f, q.codes, q.scales, 1, 1.0, bias, y, tile_e, tile_r, num, bn, ops.status, *((1.702, 7.0, 512.0) if glu else ()))
    dense = q.dense().double()
    for i, (e, _) in enumerate(tiles):
        s = slice(i * bn, (i + 1) * bn)
        ref = x[s].double() @ dense[e].t() + bias[e].double()
        if glu:
            g, u = ref[:, 0::2].clamp(max=7.0), ref[:, 1::2].clamp(-7.0, 7.0)
            ref = g * torch.sigmoid(1.702 * g) * (u + 1) * 512.0
        # 0.05 x sqrt(k) in front of the activation; its fp16 result is rounded to 2^-11
        assert _rel(y[s][real[s]], ref[real[s]]) < 2.5e-3
    assert ops.check_status() == 0
