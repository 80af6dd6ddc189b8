"""Kernels of a step at the edges of their tiles and rules: CTA-pair products over splits of K, block-FP8 products of both tile widths,
rotation of prompt rows, widened logits, and given steps queued without waiting for one another."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fllm_b200.ops import get_ops
    return get_ops(torch.device("cuda:0"))


def _rand(shape, seed, std=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std).to(torch.bfloat16).cuda()


def _rel(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("T", [129, 200, 255, 256, 257, 511])
@pytest.mark.parametrize("N,K", [(256, 4096), (264, 64), (1000, 320), (6144, 4096), (4096, 12288)])
def test_pairs_over_splits(ops, T, N, K):
    """One rounding to bf16 is all that a correct product is off (0.17 % in the mean square)."""
    x, w, b = _rand((T, K), 1), _rand((N, K), 2, 0.05), _rand((N,), 3)
    ref = x.double() @ w.double().t()
    assert _rel(ops.linear(x, w), ref) < 2.5e-3
    assert _rel(ops.linear(x, w, b), ref + b.double()) < 2.5e-3
    assert ops.check_status() == 0


@pytest.mark.parametrize("T", [129, 200, 255, 257, 511])
@pytest.mark.parametrize("N,K", [(256, 4096), (264, 64), (1000, 320), (4096, 1088)])
def test_pair_kernel_over_each_number_of_splits(ops, T, N, K):
    """The kernel itself, whatever the planner picks: an unsplit product is off by one rounding, fp32 sums over parts of K by none."""
    x, w, b = _rand((T, K), 1), _rand((N, K), 2, 0.05), _rand((N,), 3)
    ref = x.double() @ w.double().t()
    y = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    assert ops.k.linear_pair(x, w, b, y, ops.status) == 1
    assert _rel(y, ref + b.double()) < 2.5e-3
    for splits in (2, 3, 8):
        part = torch.full((splits + 1, T, N), 7.0, device="cuda")
        n = ops.k.linear_pair(x, w, None, y, ops.status, splits, part[:splits])
        assert 1 <= n <= splits and (part[n if n > 1 else 0:] == 7.0).all()
        assert n == 1 or _rel(part[:n].double().sum(0), ref) < 1e-5
    with pytest.raises(RuntimeError, match="partials"):
        ops.k.linear_pair(x, w, None, y, ops.status, 2, None)
    assert ops.check_status() == 0


@pytest.mark.parametrize("T", [129, 256, 300])
@pytest.mark.parametrize("N,K", [(256, 64), (264, 320), (1000, 1088)])
@pytest.mark.parametrize("width", [32, 96, 160, 224])
def test_pair_kernel_of_each_width(ops, T, N, K, width):
    """Tiles that end in the middle of the features, of a box and of a block of 32: one rounding, and nothing beyond the rows."""
    x, w, b = _rand((T, K), 1), _rand((N, K), 2, 0.05), _rand((N,), 3)
    ref = x.double() @ w.double().t()
    y = torch.full((T + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    assert ops.k.linear_pair(x, w, b, y[:T], ops.status, 1, None, width) == 1
    assert _rel(y[:T], ref + b.double()) < 2.5e-3 and (y[T] == 7.0).all()
    part = torch.full((3, T, N), 7.0, device="cuda")
    n = ops.k.linear_pair(x, w, None, y[:T], ops.status, 2, part[:2], width)
    assert (part[n if n > 1 else 0:] == 7.0).all() and (n == 1 or _rel(part[:n].double().sum(0), ref) < 1e-5)
    with pytest.raises(RuntimeError, match="multiple of 32"):
        ops.k.linear_pair(x, w, None, y[:T], ops.status, 1, None, width + 8)
    assert ops.check_status() == 0


@pytest.mark.parametrize("T", [129, 200, 300])
def test_pairs_leave_their_sums_to_the_norm_and_the_activation(ops, T):
    x, w, b, nw = _rand((T, 4096), 1), _rand((4096, 4096), 2, 0.02), _rand((4096,), 3), _rand((4096,), 4)
    res = _rand((T, 4096), 5)
    y = ops.linear(x, w, b, defer=True)
    assert type(y).__name__ == "Deferred"
    a, r1 = res.clone(), res.clone()
    got = ops.rmsnorm(a, y, nw, 1e-6)
    want = ops.rmsnorm(r1, ops.linear(x, w, b), nw, 1e-6)
    assert torch.equal(a, r1) and _rel(got, want.double()) < 1e-3      # (the two norms add a row's squares in other orders)
    g = _rand((2048, 512), 6, 0.1)                     # gate | up in blocks of 16
    h = _rand((T, 512), 7)
    u = (h.double() @ g.double().t()).view(T, 64, 2, 16)
    ref = (torch.nn.functional.silu(u[:, :, 0]) * u[:, :, 1]).reshape(T, 1024)
    assert _rel(ops.linear_glu(h, g, None, 0, layout=16), ref) < 2.5e-3


@pytest.mark.parametrize("T,N,K", [(200, 4768, 4096), (5, 2048, 4096), (129, 2048, 512), (512, 2336, 4096)])
@pytest.mark.parametrize("kind,layout", [(0, 16), (1, 16), (2, 0)])
def test_gate_and_up_sums_stay_in_fp32(ops, T, N, K, kind, layout):
    """A product over splits of K feeds the activation its fp32 sums: one rounding to bf16, behind the activation."""
    w, h, b = _rand((N, K), 6, 0.02), _rand((T, K), 7), _rand((N,), 8, 0.3)
    y = torch.empty(T, N // 2, dtype=torch.bfloat16, device="cuda")
    ref = h.double() @ w.double().t() + b.double()
    u = ref.view(T, N // 32, 2, 16) if layout else ref.view(T, N // 2, 2)
    gate, up = (u[:, :, 0], u[:, :, 1]) if layout else (u[..., 0], u[..., 1])
    if kind == 2:
        gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
        want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    else:
        want = (torch.nn.functional.silu(gate) if kind == 0 else torch.nn.functional.gelu(gate, approximate="tanh")) * up
    _, splits = ops.k.linear_ex(h, w, b, y, ops.workspace, ops.status, 2, kind + 1, 16 if layout else 1, 1.702, 7.0, True)
    assert splits == 2
    ops.k.glu_ex(None, y, kind, 1.702, 7.0, layout, ops.workspace, splits, b)
    assert _rel(y, want.reshape(T, N // 2)) < 2.5e-3
    assert _rel(ops.linear_glu(h, w, b, kind, 1.702, 7.0, layout), want.reshape(T, N // 2)) < 2.5e-3
    assert ops.check_status() == 0


@pytest.mark.parametrize("T,N,K", [(1, 128, 128), (17, 256, 1024), (64, 384, 8192), (65, 128, 256), (128, 7168, 8192), (129, 1280, 8192), (128, 256, 12288),
                                   (300, 8192, 1024), (513, 1280, 8192), (100, 8192, 384), (257, 512, 128), (1965, 1280, 8192), (2430, 2048, 1024), (1965, 8192, 3584)])
def test_fp8_block(ops, T, N, K):
    from fllm_b200.ops.native import Fp8BlockLinear, quantize_weight_fp8_block
    x, bias = _rand((T, K), 1), _rand((N,), 3)
    wq, sw = quantize_weight_fp8_block(_rand((N, K), 2, 0.05))
    xq, sx = torch.empty(T, K, dtype=torch.uint8, device="cuda"), torch.empty(T, K // 128, device="cuda")
    ops.k.quant_fp8_1x128(x, xq, sx)
    amax = x.float().view(T, K // 128, 128).abs().amax(-1)
    assert torch.allclose(sx, amax / 448.0, rtol=1e-6)
    xd = xq.view(torch.float8_e4m3fn).double().view(T, K // 128, 128) * sx.double()[:, :, None]
    assert ((xd.view(T, K) - x.double()).abs() <= x.double().abs() / 15.9 + sx.double().repeat_interleave(128, 1) * 2.0 ** -10).all()
    wd = wq.view(torch.float8_e4m3fn).double().view(N // 128, 128, K // 128, 128) * sw.double()[:, None, :, None]
    ref = xd.view(T, K) @ wd.view(N, K).t() + bias.double()
    assert _rel(Fp8BlockLinear(ops, wq, sw, bias)(x), ref) < 2.5e-3
    out = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    from fllm_b200.ops.native import Fp8BlockWeight
    assert ops.linear(x, Fp8BlockWeight(wq, sw), bias, out=out) is out and _rel(out, ref) < 2.5e-3
    assert ops.check_status() == 0


@pytest.mark.parametrize("T,N,K", [(1, 19072, 256), (16, 18944, 512), (16, 19072, 512), (13, 38016, 1152), (9, 7168, 8192), (16, 8192, 28672), (17, 19072, 512)])
def test_fp8_block_of_few_tokens_over_more_tiles_than_sms(ops, T, N, K):
    """Up to 16 tokens: on both sides of the number of tiles from which two CTAs share an SM, with and without splits."""
    from fllm_b200.ops.native import Fp8BlockLinear, quantize_weight_fp8_block
    x, bias = _rand((T, K), 1), _rand((N,), 3)
    wq, sw = quantize_weight_fp8_block(_rand((N, K), 2, 0.05))
    xq, sx = torch.empty(T, K, dtype=torch.uint8, device="cuda"), torch.empty(T, K // 128, device="cuda")
    ops.k.quant_fp8_1x128(x, xq, sx)
    xd = (xq.view(torch.float8_e4m3fn).double().view(T, K // 128, 128) * sx.double()[:, :, None]).view(T, K)
    wd = (wq.view(torch.float8_e4m3fn).float().view(N // 128, 128, K // 128, 128) * sw[:, None, :, None]).view(N, K)
    ref = xd @ wd.double().t() + bias.double()
    y = Fp8BlockLinear(ops, wq, sw, bias)(x)
    assert _rel(y, ref) < 2.5e-3 and max(_rel(y[t], ref[t]) for t in range(T)) < 2.8e-3
    assert ops.check_status() == 0


@pytest.mark.parametrize("T,N,K,room", [(2048, 8192, 14336, None), (800, 8192, 28672, None), (65, 256, 8320, 0), (300, 384, 12288, 0), (257, 256, 32768, 0)])
def test_fp8_block_of_many_tokens_needs_no_room_for_deep_sums(ops, T, N, K, room):
    """More than 64 tokens read their scales from global memory: K is not limited by what a workspace holds."""
    from fllm_b200.ops.native import quantize_weight_fp8_block
    x = _rand((T, K), 1)
    wq, sw = quantize_weight_fp8_block(_rand((N, K), 2, 0.05))
    xq, sx = torch.empty(T, K, dtype=torch.uint8, device="cuda"), torch.empty(T, K // 128, device="cuda")
    ops.k.quant_fp8_1x128(x, xq, sx)
    y = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    ops.k.linear_fp8_block(xq, sx, wq, sw, None, y, ops.status, ops.workspace if room is None else None)
    xd = (xq.view(torch.float8_e4m3fn).double().view(T, K // 128, 128) * sx.double()[:, :, None]).view(T, K)
    for n in range(0, N, 1024):                          # (fp64 copies of a slice of the weights at a time)
        w, s = wq[n:n + 1024], sw[n // 128:(n + 1024) // 128]
        wd = w.view(torch.float8_e4m3fn).double().view(-1, 128, K // 128, 128) * s.double()[:, None, :, None]
        assert _rel(y[:, n:n + 1024], xd @ wd.view(-1, K).t()) < 2.5e-3
    assert ops.check_status() == 0


@pytest.mark.parametrize("T,N,K", [(8, 19072, 4096), (20, 19072, 4096), (64, 19072, 5120), (3, 256, 1024)])
def test_fp8_block_into_rows_of_four_bytes(ops, T, N, K):
    """Rows that the kernels adding partial sums could not store are not split; what no kernel could store is refused."""
    from fllm_b200.ops.native import Fp8BlockWeight, quantize_weight_fp8_block
    x, w = _rand((T, K), 1), Fp8BlockWeight(*quantize_weight_fp8_block(_rand((N, K), 2, 0.05)))
    want = ops.linear(x, w)
    out = torch.zeros(T, N + 6, dtype=torch.bfloat16, device="cuda")
    ops.linear(x, w, out=out[:, 2:2 + N])
    # (two results, each off by one rounding to bf16: 0.17 % in the mean square)
    assert _rel(out[:, 2:2 + N], want.double()) < 3.4e-3 and not out[:, :2].any() and not out[:, 2 + N:].any()
    with pytest.raises(RuntimeError, match="aligned"):
        ops.linear(x, w, out=out[:, 1:1 + N])
    wide = _rand((65, K), 1)
    with pytest.raises(RuntimeError, match="aligned"):
        ops.linear(wide, w, out=torch.zeros(65, N + 6, dtype=torch.bfloat16, device="cuda")[:, 2:2 + N])


@pytest.mark.parametrize("T,N,K", [(65, 7168, 8192), (128, 1280, 8192), (300, 2048, 1024), (1000, 7168, 256)])
def test_fp8_block_of_many_tokens_into_rows_of_eight_bytes(ops, T, N, K):
    """Stored by the kernel that adds partial sums, four features at a time; where there is no room for them, refused."""
    from fllm_b200.ops.native import Fp8BlockWeight, quantize_weight_fp8_block
    x, w = _rand((T, K), 1), Fp8BlockWeight(*quantize_weight_fp8_block(_rand((N, K), 2, 0.05)))
    want = ops.linear(x, w)
    out = torch.zeros(T, N + 12, dtype=torch.bfloat16, device="cuda")
    ops.linear(x, w, out=out[:, 4:4 + N])
    assert _rel(out[:, 4:4 + N], want.double()) < 3.4e-3 and not out[:, :4].any() and not out[:, 4 + N:].any()     # (one rounding each)
    xq, sx = torch.empty(T, K, dtype=torch.uint8, device="cuda"), torch.empty(T, K // 128, device="cuda")
    ops.k.quant_fp8_1x128(x, xq, sx)
    with pytest.raises(RuntimeError, match="aligned"):
        ops.k.linear_fp8_block(xq, sx, w.wq, w.sw, None, out[:, 4:4 + N], ops.status, None)
    assert ops.check_status() == 0


@pytest.mark.parametrize("T", [147, 148, 301])
@pytest.mark.parametrize("D,hq,hkv", [(64, 5, 1), (64, 64, 8), (128, 3, 3), (128, 32, 8)])
@pytest.mark.parametrize("norm", [False, True])
def test_rope_of_prompt_rows(ops, T, D, hq, hkv, norm):
    """On both sides of the number of tokens that the kernel for rows takes over at, against the PyTorch operator."""
    from fllm_b200.ops.reference import RefOps
    qkv = _rand((T, (hq + 2 * hkv) * D), 1)
    blocks = T // 16 + 2
    pos = (torch.arange(T) * 37 % 9000).int().cuda()
    slots = torch.randperm(blocks * 16, generator=torch.Generator().manual_seed(2))[:T].int().cuda()
    slots[3], slots[T - 1] = -1, -1
    inv = (1e6 ** (-torch.arange(0, D, 2).double() / D)).float().cuda()
    qn, kn = (_rand((D,), 3) + 1, _rand((D,), 4) + 1) if norm else (None, None)
    caches = [[torch.zeros(blocks, hkv, 16, D, dtype=torch.bfloat16, device="cuda") for _ in range(2)] for _ in range(2)]
    got = ops.rope_kv_write(qkv.clone(), pos, slots, inv, qn, kn, *caches[0], hq, hkv, D, D, 0, 1e-6, 1.25)
    want = RefOps().rope_kv_write(qkv.clone(), pos, slots, inv, qn, kn, *caches[1], hq, hkv, D, D, 0, 1e-6, 1.25)
    # one rounding to bf16 more or less, and one of a normed value
    assert _rel(got, want.double()) < 4e-3 and _rel(caches[0][0], caches[1][0].double()) < 4e-3
    assert torch.equal(caches[0][1], caches[1][1])


@pytest.mark.parametrize("rows,cols,pitch", [(1, 1, 8), (3, 7, 8), (5, 4096, 4096), (2, 151936, 151936), (4, 2052, 2056), (3, 2051, 2056)])
def test_widen_rows(ops, rows, cols, pitch):
    x = _rand((rows, pitch), 1)[:, :cols]
    assert torch.equal(ops.widen_rows(x), x.float())


def test_given_steps_queue_without_waiting():
    """Steps of other sizes and other tokens, one after the other without a synchronisation: each gives what it gives alone."""
    from fllm_b200.config import EngineConfig, preset
    from fllm_b200.runtime import LLMEngine
    from fllm_b200.runtime.request import Request, SamplingParams
    from fllm_b200.runtime.scheduler import ScheduledSeq, ScheduledStep
    cfg = preset("qwen3-tiny")
    eng = LLMEngine(cfg, EngineConfig(max_num_seqs=16, max_num_batched_tokens=128, max_model_len=256, num_kv_blocks=256, enable_prefix_caching=False),
                    device="cuda:0")
    g = torch.Generator().manual_seed(0)
    reqs = []
    for i in range(11):
        toks = torch.randint(0, cfg.vocab_size, (9 + 5 * i,), generator=g).tolist()
        r = Request(f"r{i}", 1000 + i, toks, SamplingParams(max_tokens=4))
        r.output = [7 + i]
        eng.blocks.allocate(r.seq_id, [])
        assert eng.blocks.ensure_capacity(r.seq_id, r.num_tokens)
        reqs.append(r)
    prompts = [ScheduledStep(seqs=[ScheduledSeq(r, 0, len(r.prompt), True)]) for r in reqs]
    decodes = [ScheduledStep(seqs=[ScheduledSeq(r, len(r.prompt), 1, j % 3 != 1) for j, r in enumerate(reqs[a:b])]) for a, b in ((0, 11), (2, 5), (4, 11), (0, 1), (3, 11))]
    alone = []
    for s in prompts + decodes:
        alone.append(eng.run_forced(s).cpu())
        torch.cuda.synchronize()
    queued = [eng.run_forced(s) for s in prompts + decodes + decodes[::-1]]
    torch.cuda.synchronize()
    for a, b in zip(alone + alone[len(prompts):][::-1], queued):
        assert torch.equal(a, b.cpu())
    # from streams that know nothing of one another: each step waits for the one before, wherever that was queued
    streams, spread = [torch.cuda.Stream() for _ in range(2)], []
    for i, s in enumerate(prompts + decodes):
        with torch.cuda.stream(streams[i % 2]):
            spread.append(eng.run_forced(s))
    torch.cuda.synchronize()
    for a, b in zip(alone, spread):
        assert torch.equal(a, b.cpu())
    eng.close()


@pytest.mark.parametrize("D,hq,hkv,window", [(128, 32, 8, 0), (64, 32, 8, 0), (128, 32, 8, 70)])
@pytest.mark.parametrize("kv", [(320, 257, 65, 64), (333, 300, 129, 1), (449, 448, 447, 385)])
def test_prompt_attention_rescales_between_halves(ops, D, hq, hkv, window, kv):
    """Scores that grow along the sequence move the row maximum by more than 2^8 in every half tile of 64 tokens, the last of which may
    be the first half of a tile. Probabilities and results are rounded to bf16 once each: 2^-9 + 2^-9."""
    from types import SimpleNamespace
    G, n = hq // hkv, len(kv)
    starts = [0]
    for x in kv:
        starts.append(starts[-1] + x)
    per = [(x + 15) // 16 for x in kv]
    tables = torch.zeros(n, max(per), dtype=torch.int32, device="cuda")
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(1)).int().cuda()
    kc, vc = torch.zeros(sum(per), hkv, 16, D, dtype=torch.bfloat16, device="cuda"), _rand((sum(per), hkv, 16, D), 2)
    q = (_rand((starts[-1], hq * D), 3, 0.2).float() + 1).to(torch.bfloat16)
    ref, o = [], 0
    for i, x in enumerate(kv):
        blocks = order[o:o + per[i]]
        o += per[i]
        tables[i, :per[i]] = blocks
        k = _rand((per[i] * 16, hkv, D), 4 + i, 0.2).float() + (torch.arange(per[i] * 16, device="cuda") / 8 * D ** -0.5)[:, None, None]
        kc[blocks.long()] = k.to(torch.bfloat16).view(per[i], 16, hkv, D).transpose(1, 2)
        k, v = (c[blocks.long()].double().transpose(1, 2).reshape(-1, hkv, D)[:x].repeat_interleave(G, 1) for c in (kc, vc))
        s = torch.einsum("qhd,khd->hqk", q[starts[i]:starts[i + 1]].double().view(x, hq, D), k) * D ** -0.5
        d = torch.arange(x, device="cuda")[:, None] - torch.arange(x, device="cuda")[None, :]
        s = s.masked_fill((d < 0) | ((d >= window) if window else (d < 0)), float("-inf"))
        ref.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v).reshape(x, hq * D))
    i32 = dict(dtype=torch.int32, device="cuda")
    rows = torch.tensor([i for i, x in enumerate(kv) for _ in range(x)], **i32)
    pos = torch.tensor([j for x in kv for j in range(x)], **i32)
    meta = SimpleNamespace(q_starts=torch.tensor(starts, **i32), seq_lens=torch.tensor(kv, **i32), num_seqs=n, max_q_len=max(kv),
                           min_q_len=min(kv), max_kv_len=max(kv))
    y = ops.attention(q, kc, vc, tables, rows, pos, hq, hkv, D, D ** -0.5, window, None, 0.0, meta=meta)
    assert _rel(y, torch.cat(ref)) < 2 ** -8
    assert ops.check_status() == 0


def _attention(ops, q_lens, kv_lens, D, hq, hkv, window, softcap=0.0, sinks=False, seed=1, longest=0):
    """Paged attention of sequences whose last q_lens tokens are queries -> (kernel's result, the same in 64 bits)."""
    from types import SimpleNamespace
    G, n = hq // hkv, len(kv_lens)
    per = [(x + 15) // 16 for x in kv_lens]
    tables = torch.zeros(n, max(per), dtype=torch.int32, device="cuda")
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(seed)).int().cuda()
    kc, vc, q = _rand((sum(per), hkv, 16, D), seed + 1), _rand((sum(per), hkv, 16, D), seed + 2), _rand((sum(q_lens), hq * D), seed + 3)
    sk = _rand((hq,), seed + 4).float() if sinks else None
    starts, ref, o = [0], [], 0
    for m, x, b in zip(q_lens, kv_lens, per):
        blocks = order[o:o + b]
        tables[len(starts) - 1, :b] = blocks
        o += b
        k, v = (c[blocks.long()].double().transpose(1, 2).reshape(-1, hkv, D)[:x].repeat_interleave(G, 1) for c in (kc, vc))
        s = torch.einsum("qhd,khd->hqk", q[starts[-1]:starts[-1] + m].double().view(m, hq, D), k) * D ** -0.5
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        d = torch.arange(x - m, x, device="cuda")[:, None] - torch.arange(x, device="cuda")[None, :]
        s = s.masked_fill((d < 0) | ((d >= window) if window else (d < 0)), float("-inf"))
        if sinks:
            s = torch.cat([s, sk.double()[:, None, None].expand(hq, m, 1)], -1)
        p = torch.softmax(s, -1)[..., :x]
        ref.append(torch.einsum("hqk,khd->qhd", p, v).reshape(m, hq * D))
        starts.append(starts[-1] + m)
    i32 = dict(dtype=torch.int32, device="cuda")
    meta = SimpleNamespace(q_starts=torch.tensor(starts, **i32), seq_lens=torch.tensor(kv_lens, **i32), num_seqs=n, max_q_len=max(longest, *q_lens),
                           min_q_len=min(q_lens), max_kv_len=max(kv_lens))
    rows = torch.tensor([i for i, m in enumerate(q_lens) for _ in range(m)], **i32)
    pos = torch.tensor([x - m + j for m, x in zip(q_lens, kv_lens) for j in range(m)], **i32)
    y = ops.attention(q, kc, vc, tables, rows, pos, hq, hkv, D, D ** -0.5, window, sk, softcap, meta=meta)
    assert ops.check_status() == 0
    return y, torch.cat(ref)


@pytest.mark.parametrize("D,hq,hkv", [(128, 32, 8), (64, 64, 8)])
@pytest.mark.parametrize("window", [1, 127, 128, 129, 159, 160, 161, 191, 192, 193, 256, 300, 511, 2000])
@pytest.mark.parametrize("sinks", [False, True])
def test_prompt_attention_under_windows(ops, D, hq, hkv, window, sinks):
    """Windows around the tiles of 128 keys and the 32 and 64 queries of a tile: tiles that every row sees whole, and those at both edges.
    Probabilities and results are rounded to bf16 once each: 2^-9 + 2^-9."""
    y, ref = _attention(ops, (700, 513, 1, 300), (700, 1100, 400, 333), D, hq, hkv, window, sinks=sinks)
    assert _rel(y, ref) < 2 ** -8


@pytest.mark.parametrize("D,hq,hkv", [(128, 16, 16), (64, 32, 16), (128, 32, 2), (64, 64, 8)])
@pytest.mark.parametrize("window", [0, 255, 256])
@pytest.mark.parametrize("q_lens,kv_lens", [((1291, 1291), (1291, 1500)), ((1301, 40), (1307, 50)), ((129, 3), (260, 3))])
def test_prompt_attention_over_groups_and_ragged_tiles(ops, D, hq, hkv, window, q_lens, kv_lens):
    """Groups of 1, 2, 8 and 16 query heads, last tiles of a few rows, and windows on both sides of two tiles of keys, where one or two tiles
    of queries share a block. Probabilities and results are rounded to bf16 once each: 2^-9 + 2^-9."""
    y, ref = _attention(ops, q_lens, kv_lens, D, hq, hkv, window)
    assert _rel(y, ref) < 2 ** -8


@pytest.mark.parametrize("D,hq,hkv,window", [(128, 32, 8, 0), (64, 64, 8, 128), (64, 32, 8, 0), (128, 16, 16, 100)])
@pytest.mark.parametrize("q_lens", [[1] * 40 + [300], [300] + [1] * 40, [1, 2, 700, 1, 64, 1, 1, 129, 1], [1] * 500 + [40], [1] * 3 + [1000, 1000] + [2] * 200])
def test_decode_rows_beside_prompts(ops, D, hq, hkv, window, q_lens):
    """Many decode rows and a few prompts in one call, in any order: every row is written, none by another's tile."""
    kv = [m + (i * 37) % 300 for i, m in enumerate(q_lens)]
    y, ref = _attention(ops, q_lens, kv, D, hq, hkv, window)
    o = 0
    for m in q_lens:
        assert _rel(y[o:o + m], ref[o:o + m]) < 2 ** -7     # (a single row: twice the mean square of all)
        o += m
    assert _rel(y, ref) < 2 ** -8


@pytest.mark.parametrize("q_lens", [[1], [1, 2], [1, 2, 7]])
def test_longest_prompt_given_as_an_upper_bound(ops, q_lens):
    """Fewer rows in all than the shortest prompt has: the prompt kernel finds nothing or one sequence, the decode kernel does the rest."""
    y, ref = _attention(ops, q_lens, [m + 50 for m in q_lens], 128, 32, 8, 0, longest=64)
    assert _rel(y, ref) < 2 ** -7


def _planes(S, rows, cols, seed):
    """Workspace with S planes of partial sums, and their sum in the order of the planes."""
    p = (torch.randn(S, rows, cols, generator=torch.Generator().manual_seed(seed))).cuda()
    ws = torch.zeros(65536 + p.numel() * 4, dtype=torch.uint8, device="cuda")
    ws[65536:].view(torch.float32).copy_(p.view(-1))
    total = p[0].clone()
    for s in range(1, S):
        total += p[s]
    return ws, total


@pytest.mark.parametrize("D,hq,hkv", [(64, 6, 2), (128, 8, 1), (256, 2, 1)])
@pytest.mark.parametrize("S", [2, 4, 5, 6, 9])
@pytest.mark.parametrize("T", [3, 300])
def test_rotation_adds_planes_in_either_way(ops, D, hq, hkv, S, T):
    """Few and many rows, planes on both sides of a batch: the bits of the rotation of the summed projection."""
    ws, total = _planes(S, T, (hq + 2 * hkv) * D, S)
    bias, w = _rand(((hq + 2 * hkv) * D,), 3), _rand((D,), 4)
    pos = torch.arange(T, dtype=torch.int32, device="cuda")
    inv = (1e4 ** (-torch.arange(0, D, 2, device="cuda").float() / D)).contiguous()
    caches = [torch.zeros(-(-T // 16), hkv, 16, D, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    q = torch.empty(T, hq * D, dtype=torch.bfloat16, device="cuda")
    ops.k.rope_kv_write_splitk(ws, S, bias, q, pos, pos, inv, w, w, *caches[:2], hq, hkv, D, D, 1, 1e-6, 1.0)
    qkv = (total + bias.float()).to(torch.bfloat16)
    ops.k.rope_kv_write(qkv, pos, pos, inv, w, w, *caches[2:], hq, hkv, D, D, 1, 1e-6, 1.0)
    assert torch.equal(q, qkv[:, :hq * D]) and torch.equal(caches[0], caches[2]) and torch.equal(caches[1], caches[3])


@pytest.mark.parametrize("H", [512, 2048, 4096])
@pytest.mark.parametrize("S", [2, 4, 9])
@pytest.mark.parametrize("T", [1, 148, 149, 300])
def test_norm_adds_planes_in_either_way(ops, H, S, T):
    """Rows on both sides of what the SMs hold at once: the bits of the norm of the summed product."""
    ws, total = _planes(S, T, H, S)
    w, r = _rand((H,), 4), _rand((T, H), 5)
    r2, y, y2 = r.clone(), torch.empty_like(r), torch.empty_like(r)
    ops.k.rmsnorm_splitk(r, ws, S, None, w, y, 1e-6, 0.0)
    ops.k.rmsnorm(r2, total.to(torch.bfloat16), w, y2, 1e-6, 0.0)
    assert torch.equal(r, r2) and _rel(y, y2.double()) < 1e-3        # (the sum of squares in another order: a last bit here and there)


@pytest.mark.parametrize("act,layout", [(0, 16), (1, 0), (2, 0)])
@pytest.mark.parametrize("T,S", [(1, 2), (50, 2), (50, 6), (200, 2), (200, 3)])
def test_activation_adds_planes_in_either_way(ops, act, layout, T, S):
    """Few, some and many blocks: one rounding to bf16 behind fp32 sums."""
    I = 4096
    ws, total = _planes(S, T, 2 * I, S)
    y = torch.empty(T, I, dtype=torch.bfloat16, device="cuda")
    ops.k.glu_ex(None, y, act, 1.702, 7.0, layout, ws, S, None)
    x = total.double()
    if layout == 16:
        x = x.view(T, I // 16, 2, 16)
        g, u = x[:, :, 0].reshape(T, I), x[:, :, 1].reshape(T, I)
    else:
        g, u = (x[:, 0::2], x[:, 1::2]) if act == 2 else (x[:, :I], x[:, I:])
    if act == 2:
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        ref = g * torch.sigmoid(1.702 * g) * (u + 1)
    else:
        ref = (torch.nn.functional.silu(g) if act == 0 else torch.nn.functional.gelu(g, approximate="tanh")) * u
    assert _rel(y, ref) < 2.5e-3


@pytest.mark.parametrize("T,S", [(16, 8), (100, 8), (100, 5), (256, 9)])
def test_product_adds_planes_in_either_way(ops, T, S):
    """Fewer and more blocks than SMs, planes on both sides of a batch: the bits of the planes added in their order."""
    x, w, b = _rand((T, 2304), 1), _rand((2048, 2304), 2, 0.05), _rand((2048,), 3)
    y = torch.empty(T, 2048, dtype=torch.bfloat16, device="cuda")
    ops.k.linear(x, w, b, y, ops.workspace, ops.status, S)
    n = T * 2048
    p = ops.workspace[65536:65536 + S * n * 4].view(torch.float32).view(S, T, 2048)
    total = p[0].clone()
    for s in range(1, S):
        total += p[s]
    assert torch.equal(y, (total + b.float()).to(torch.bfloat16)) and _rel(y, x.double() @ w.double().t() + b.double()) < 2.5e-3
    assert ops.check_status() == 0
