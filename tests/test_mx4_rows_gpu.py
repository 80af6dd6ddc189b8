"""MXFP4 expert stacks on the block-scaled tensor cores: rows as sums of e4m3 pieces, grouped products at the edges of tiles."""
import pytest
import torch

from fllm_b200.ops.fp4 import Fp4ExpertStack, scale_atoms


@pytest.fixture(scope="module")
def ops():
    from fllm_b200.ops import get_ops
    return get_ops(torch.device("cuda:0"))


def _rand(shape, seed, std=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std).to(torch.bfloat16)


def _rel(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


def _room(rows, n, bn, pieces, fill=0xFF):
    """Pieces and scale atoms, filled with what is not a number: whatever a product reads has been written."""
    full = lambda *shape: torch.full(shape, fill, dtype=torch.uint8, device="cuda")
    return full(rows * pieces, n), full(rows // bn * -(-n // 128) * -(-bn * pieces // 128), 512)


def _values(q, sf, bn, pieces):
    """[rows, k] in 64 bits of the sums of pieces."""
    rows, k = q.shape[0] // pieces, q.shape[1]
    kb, atoms = -(-k // 128), -(-bn * pieces // 128)
    s = sf.view(rows // bn, kb, atoms, 32, 4, 4).permute(0, 2, 4, 3, 1, 5).reshape(rows // bn, atoms * 128, kb * 4)[:, :bn * pieces, :k // 32]
    v = q.view(torch.float8_e4m3fn).double().view(rows // bn, bn * pieces, k // 32, 32)
    s = torch.where(s == 255, float("nan"), torch.exp2(s.double() - 127))
    return (v * s[..., None]).view(rows // bn, bn // 16, pieces, 16, k).sum(2).view(rows, k).cpu()


def test_scale_atoms_hold_every_scale():
    s = torch.randint(0, 255, (2, 200, 6), dtype=torch.uint8, generator=torch.Generator().manual_seed(1))
    a = scale_atoms(s)
    assert a.shape == (2, 2, 2, 512)
    for e, n, g in ((0, 0, 0), (1, 127, 3), (0, 128, 4), (1, 199, 5), (1, 45, 2)):
        r = n % 128
        assert a[e, n // 128, g // 4, (r % 32) * 16 + (r // 32) * 4 + g % 4] == s[e, n, g]
    assert a[0, 1, 0, (100 % 32) * 16 + (100 // 32) * 4] == 127 and a[0, 0, 1, 2] == 127


def test_bytes_of_a_stack_count_its_atoms():
    from types import SimpleNamespace
    from fllm_b200.comm.ep_a2a import release_scale_atoms
    s = Fp4ExpertStack.from_dense(_rand((2, 128, 192), 3))
    plain = 2 * 128 * 96 + 2 * 128 * 6
    assert s.atoms is None and s.nbytes() == plain
    s.atoms = scale_atoms(s.scales)
    assert s.nbytes() == plain + 2 * 1 * 2 * 512
    release_scale_atoms([SimpleNamespace(exp_gate_up=s, exp_down=torch.empty(1)), SimpleNamespace(exp_gate_up=None, exp_down=None)])
    assert s.atoms is None and s.nbytes() == plain


@pytest.mark.gpu
def test_stacks_reach_the_gpu_in_one_copy():
    """K ends in the middle of a block: the bytes behind the codes are there from the start. Codes, a sixteenth of them in scales, as much in
    atoms and in what these are made from; a second copy of the codes would be another whole."""
    s = Fp4ExpertStack.from_dense(_rand((4, 2048, 1984), 3))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    g = s.to("cuda")
    assert torch.cuda.max_memory_allocated() - before < 1.6 * s.codes.numel()
    assert g.atoms is not None and torch.equal(g.codes.cpu(), s.codes) and g.codes.untyped_storage().nbytes() == s.codes.numel() + 32


@pytest.mark.gpu
@pytest.mark.parametrize("bn", [16, 32, 80])
@pytest.mark.parametrize("K", [64, 320, 2880, 8192])
def test_rows_are_the_sum_of_their_pieces(ops, K, bn):
    """Exact down to 2^-12 of the largest of a block of 32 (top): what the first piece leaves of it is 2^-4 top at most, so the second piece's
    scale is 2^-4 top / 224 at most and its smallest step 2^-9 of that, 2^-20.8 top, while 8 bits of a value from 2^-12 top on end at 2^-19 top. Smaller
    values may be off by half of that step. Blocks with an infinity or a NaN are not numbers; other rows and blocks are."""
    x = _rand((9, K), 1)
    x[0] *= 2.0 ** 100
    x[1] *= 2.0 ** -90
    x[2] = 0
    x[3, 1::2] *= 2.0 ** -13
    x[4, 5], x[5, 6], x[5, 7] = float("nan"), float("inf"), -float("inf")
    x[6] = torch.finfo(torch.bfloat16).max
    x[7, ::3] *= 2.0 ** -20
    rows = -(-20 // bn) * bn
    token_of = torch.full((rows,), -1, dtype=torch.int32)
    at = list(range(8)) if bn == 16 else list(range(7)) + [15]      # (groups of 16 are filled from their start)
    token_of[at] = torch.arange(8, dtype=torch.int32)
    q, sf = _room(rows, K, bn, 2)
    ops.k.moe_rows_mx(x.cuda(), token_of.cuda(), q, sf, bn)
    got, xd = _values(q, sf, bn, 2), x.double()
    for i, r in enumerate(at):
        g, w = got[r].view(-1, 32), xd[i].view(-1, 32)
        finite = w.isfinite().all(1)
        assert g[~finite].isnan().all()
        top = w[finite].abs().amax(1, keepdim=True)
        off = (g[finite] - w[finite]).abs()
        assert (off <= top * 2.0 ** -21.8).all() and (off[w[finite].abs() >= top * 2.0 ** -12] == 0).all()
    rest = [r for r in range(16) if r not in at]
    assert (got[rest] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("bn", [16, 32, 80])
@pytest.mark.parametrize("n,k", [(128, 64), (384, 192), (5760, 2880), (256, 1024)])
@pytest.mark.parametrize("glu", [False, True])
def test_grouped(ops, bn, n, k, glu):
    """Experts with no row, one, 15 to 17, a full tile and one more; the clamped activation in the epilogue, whose result feeds another
    product. A product is off by its rounding to bf16 (0.17 % in the mean square), the three pieces of an activation by 2^-12 of it and 2^-20 of the
    block's largest (fp32 exponentials and sums: 1e-6)."""
    counts = [0, 1, min(bn, 17), bn, bn + 1, 15]
    E = len(counts)
    stack = Fp4ExpertStack.from_dense(_rand((E, n, k), 3, 0.05).cuda())
    assert stack.atoms is not None
    bias = _rand((E, n), 4, 0.1).cuda()
    tiles = [(e, j) for e, c in enumerate(counts) for j in range(-(-c // bn))]
    rows = len(tiles) * bn
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    tile_e, tile_r = i32([e for e, _ in tiles] + [0] * 3), torch.arange(len(tiles) + 3, dtype=torch.int32, device="cuda") * bn
    tile_n = i32([min(bn, counts[e] - j * bn) for e, j in tiles] + [0] * 3)
    where = (tile_e, tile_r, tile_n, i32([len(tiles), rows]), bn, ops.status)
    real = torch.cat([torch.arange(bn) + j * bn < counts[e] for e, j in tiles]).cuda()
    x = _rand((rows, k), 5).cuda()
    token_of = torch.where(real, torch.arange(rows, device="cuda"), -1).int()
    q, sf = _room(rows, k, bn, 2)
    ops.k.moe_rows_mx(x, token_of, q, sf, bn)
    ref = torch.zeros(rows, n, dtype=torch.float64, device="cuda")
    dense = stack.dense().double()
    for i, (e, _) in enumerate(tiles):
        ref[i * bn:(i + 1) * bn] = x[i * bn:(i + 1) * bn].double() @ dense[e].t() + bias[e].double()
    if not glu:
        y = torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")
        ops.k.moe_grouped_linear_mx4(q, sf, 2, stack.codes, stack.atoms, 1.0, bias, y, None, *where)
        assert _rel(y[real], ref[real]) < 2.5e-3
    else:
        g, u = ref[:, 0::2].clamp(max=7.0), ref[:, 1::2].clamp(-7.0, 7.0)
        ref = g * torch.sigmoid(1.702 * g) * (u + 1)
        aq, asf = _room(rows, n // 2, bn, 3)
        ops.k.moe_grouped_linear_mx4(q, sf, 2, stack.codes, stack.atoms, 1.0, bias, aq, asf, *where, 1.702, 7.0)
        got = _values(aq, asf, bn, 3)[real.cpu()]
        assert _rel(got, ref[real].cpu()) < 2.0 ** -12
        down = Fp4ExpertStack.from_dense(_rand((E, k, n // 2), 6, 0.05).cuda())
        y = torch.empty(rows, k, dtype=torch.bfloat16, device="cuda")
        ops.k.moe_grouped_linear_mx4(aq, asf, 3, down.codes, down.atoms, 1.0, None, y, None, *where)
        ref = torch.cat([ref[i * bn:(i + 1) * bn] @ down.dense().double()[e].t() for i, (e, _) in enumerate(tiles)])
        assert _rel(y[real], ref[real]) < 2.5e-3
    assert ops.check_status() == 0


@pytest.mark.gpu
def test_rows_of_a_tile(ops):
    """moe_align counts the rows of every tile."""
    ids = torch.tensor([0] * 33 + [2] * 16 + [3], dtype=torch.int32, device="cuda").view(-1, 1)
    i32 = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")
    row_of, token_of, te, tr, tn, num = ids.clone(), i32(160), i32(10), i32(10), i32(10), i32(2)
    ops.k.moe_align(ids, 5, 0, 5, 16, row_of, token_of, te, tr, num, None, None, tn)
    assert num.tolist() == [5, 80] and te.tolist()[:5] == [0, 0, 0, 2, 3] and tn.tolist()[:5] == [16, 16, 1, 16, 1]


@pytest.mark.gpu
@pytest.mark.parametrize("bn", [16, 80])
def test_rows_that_are_in_place(ops, bn):
    """An activation between the products lies in the rows of the tiles: those with a token are converted as they are, the others of their group of 16 are zeros,
    and groups without a token stay as they were."""
    K, rows = 192, 2 * 80
    x = _rand((rows, K), 1)
    token_of = torch.full((rows,), -1, dtype=torch.int32)
    at = [0, 1, 17, 80, 95, 96] if bn == 80 else [0, 1, 80, 95]
    at = sorted({*at, *(r // 16 * 16 for r in at)})
    token_of[at] = torch.arange(len(at) - 1, -1, -1, dtype=torch.int32)          # (which token a row has does not matter here)
    x[[r for r in range(rows) if token_of[r] < 0]] = float("nan")
    q, sf = _room(rows, K, bn, 2)
    ops.k.moe_rows_mx(x.cuda(), token_of.cuda(), q, sf, bn, None, True)
    got = _values(q, sf, bn, 2)
    whole, wsf = _room(rows, K, bn, 2)
    ops.k.moe_rows_mx(x.cuda(), None, whole, wsf, bn)
    assert torch.equal(got[at], _values(whole, wsf, bn, 2)[at])
    used = {r // 16 for r in at}
    assert (got[[r for r in range(rows) if r // 16 in used and token_of[r] < 0]] == 0).all()
    pieces = q.view(rows // 16, 2 * 16, K)
    assert all((pieces[g] == 0xFF).all() for g in range(rows // 16) if g not in used)
    with pytest.raises(RuntimeError, match="as many rows"):
        ops.k.moe_rows_mx(x[:rows - 16].cuda(), token_of.cuda(), q, sf, bn, None, True)
