"""Edge sizes of the streaming kernels and of the schedule builder: remainders of their tiles, the smallest and largest
sizes of each variant, values at the ends of the formats."""
import numpy as np
import pytest
import torch

from oracle import gdpa_oracle as orc
from tests._util import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import ads_model_kernel_library_b200.gdpa as g

    return g


def _check_norm_backward(mode, rows, n, with_add, with_weight, want_dw, want_db):
    """Against autograd in fp64.  dx is a bf16 tensor: half an ulp, 2^-9 of the value; the sums in fp32 add some 1e-6 of the
    largest term.  The column sums are fp32 over `rows` terms."""
    from ads_model_kernel_library_b200.gdpa.megakernel import NORM_EPS, norm_rows_backward

    g = torch.Generator().manual_seed(rows + n)
    x, dy, add = (torch.randn(rows, 1, n, generator=g).to(torch.bfloat16) for _ in range(3))
    x = x + 0.5
    w = 1 + 0.2 * torch.randn(n, generator=g) if with_weight else torch.ones(n)
    xd, wd, bd = x.double().view(rows, n).requires_grad_(True), w.double().requires_grad_(True), torch.zeros(n).double().requires_grad_(True)
    mean = xd.mean(1, keepdim=True)
    if mode == 0:
        rstd = torch.rsqrt(xd.square().mean(1, keepdim=True) + NORM_EPS)
        y = xd * rstd * wd
    else:
        rstd = torch.rsqrt((xd - mean).square().mean(1, keepdim=True) + NORM_EPS)
        y = (xd - mean) * rstd * wd + bd
    y.backward((dy.double() + (add.double() if with_add else 0)).view(rows, n))
    dx, dw, db = norm_rows_backward(mode, dy.cuda(), add.cuda() if with_add else None, x.cuda(), w.cuda() if with_weight else None,
                                    mean.detach().float().view(-1).cuda(), rstd.detach().float().view(-1).cuda(),
                                    want_dweight=want_dw, want_dbias=want_db)
    torch.cuda.synchronize()
    ref = xd.grad.view_as(dx)
    assert ((dx.cpu().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
    assert (dw is None) == (not want_dw) and (db is None) == (not want_db)
    tol = 1e-6 * rows ** 0.5 * 16 + 1e-5  # fp32 sums of terms of a few units
    if want_dw:
        assert ((dw.cpu().double() - wd.grad).abs() <= tol * (1 + wd.grad.abs())).all()
    if want_db and mode == 1:
        assert ((db.cpu().double() - bd.grad).abs() <= tol * (1 + bd.grad.abs())).all()


@pytest.mark.parametrize("rows,n", [(1, 8), (3, 256), (37, 512), (300, 520), (1001, 1024), (29, 1032), (150, 2048), (7, 4096), (33, 4104)])
@pytest.mark.parametrize("mode", [0, 1])
def test_norm_backward_at_the_edges_of_its_row_lengths(mode, rows, n):
    """Rows of 8 ... 4104 values: one to eight warps a row, then the kernel for longer rows."""
    _check_norm_backward(mode, rows, n, mode == 1, True, n <= 4096, n <= 4096 and mode == 1)


@pytest.mark.parametrize("rows,n", [(11003, 256), (5501, 1024), (2701, 2048), (1351, 4096)])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("add,weight,dw,db", [(True, True, True, True), (False, True, True, False), (True, False, False, True)])
def test_norm_backward_over_several_rounds_of_its_grid(mode, rows, n, add, weight, dw, db):
    """Three full rounds and a part of one of 148 * 3 blocks (RMS norm; the layer norm has fewer blocks and more rounds), with
    one, two, four and eight warps a row: the column sums are carried from round to round."""
    _check_norm_backward(mode, rows, n, add, weight, dw, db and mode == 1)


@pytest.mark.parametrize("rows,n", [(30001, 8), (24001, 64), (9001, 383), (9001, 384), (500, 768), (3000, 896), (3000, 904), (700, 1536),
                                    (700, 1544), (900, 1792), (900, 1800), (300, 2560), (300, 3064), (300, 3072), (40, 8192)])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("add,weight", [(True, True), (False, False)])
def test_norm_backward_without_column_sums(mode, rows, n, add, weight):
    """On both sides of the row lengths at which the kernel changes; the first rows take several rounds of the grid."""
    _check_norm_backward(mode, rows, n // 8 * 8, add, weight, False, False)


def _schedule(qo, ko, mode, heads, max_q, max_kv, kv_index=None):
    from ads_model_kernel_library_b200.gdpa import ops

    total = int((qo if mode != 1 else ko)[-1])
    s = ops._build_schedule(mode, qo, ko, qo.numel() - 1, heads, total, max_q, max_kv, kv_index).cpu()
    return s[:4].tolist(), s[4:4 + 4 * int(s[0])].view(-1, 4)


@pytest.mark.parametrize("heads,longest", [(3, 700), (1, 120), (7, 120), (5, 20000)])
@pytest.mark.parametrize("batch", [1, 31, 1023, 1024, 1025, 2500])
@pytest.mark.parametrize("mode", [0, 1])
def test_schedule_lists_every_block_once_longest_first(mode, batch, heads, longest):
    """Some, at most four, seven and over 64 items a sequence."""
    rng = np.random.default_rng(batch)
    lq, lk = rng.integers(0, longest, batch), rng.integers(0, 4 * longest, batch)
    lq[0] = lk[0] = longest
    if longest == 20000:
        lq[batch // 2:], lk[batch // 2:] = 15000, 8000
    qo, ko = (torch.tensor(np.concatenate([[0], np.cumsum(n)])).cuda() for n in (lq, lk))
    max_q, max_kv = longest * 6 // 7, longest * 25 // 7
    header, items = _schedule(qo, ko, mode, heads, max_q, max_kv)
    tiles = lambda n, t: -(-n // t)  # noqa: E731
    cq, ck = np.minimum(lq, max_q), np.minimum(lk, max_kv)
    blocks, weight = (tiles(cq, 256), tiles(ck, 128)) if mode == 0 else (tiles(ck, 128), tiles(cq, 128))
    want = [(b, h, k, weight[b]) for b in range(batch) for h in range(heads) for k in range(blocks[b])]
    assert header[0] == header[2] == len(want) and header[1] == mode and header[3] == 0
    assert sorted(map(tuple, items.tolist())) == want
    w = items[:, 3]
    assert bool((w[1:] <= w[:-1]).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("tokens", [1, 63, 64, 129, 1000])
@pytest.mark.parametrize("shift", [0, 2])
def test_softmax_backward_for_any_number_of_tokens_and_alignment_of_the_output(D, tokens, shift):
    """rowsum(dO * O) is taken over blocks of 64 / 128 tokens, by 16-byte words where the output is aligned to them: dQ of
    the whole backward against autograd of the fp64 attention, within the bf16 bound of the kernels (2e-2)."""
    import math

    g = torch.Generator().manual_seed(tokens + D)
    H, kv = 3, 77
    q, do = (torch.randn(tokens, H, D, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    k, v = (torch.randn(kv, H, D, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    qo, ko = torch.tensor([0, tokens]).cuda(), torch.tensor([0, kv]).cuda()
    scale = 1 / math.sqrt(D)
    o, lse = torch.ops.gdpa.generalized_dot_product_attention_softmax(q, k, v, qo, ko, tokens, kv, scale)
    moved = torch.empty(o.numel() + shift, dtype=o.dtype, device="cuda")[shift:].view(o.shape).copy_(o)
    dq = torch.ops.gdpa.generalized_dot_product_attention_backward(do, q, k, v, qo, ko, tokens, kv, scale, 100, moved, lse)[0]
    torch.cuda.synchronize()
    q64 = q.double().requires_grad_(True)
    p = torch.softmax(torch.einsum("qhd,khd->hqk", q64, k.double()) * scale, -1)
    torch.einsum("hqk,khd->qhd", p, v.double()).backward(do.double())
    assert_close(dq, q64.grad, "dQ")


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("scale", [-0.1, 0.0, 0.1])
def test_softmax_forward_for_every_sign_of_the_scale(D, scale):
    """The row maximum of c * S is c times the maximum of S only for c >= 0; KV lengths at the edges of the 32- and
    64-column chunks.  Against the fp64 softmax within the bf16 bound of the kernels."""
    import ads_model_kernel_library_b200.gdpa as G

    g = torch.Generator().manual_seed(D)
    lk = [1, 31, 32, 33, 64, 65, 127, 128, 129, 400]
    lq = [1, 40, 128, 129, 300, 7, 256, 64, 200, 130]
    qo, ko = (torch.tensor(np.concatenate([[0], np.cumsum(n)])) for n in (lq, lk))
    q = (torch.randn(int(qo[-1]), 2, D, generator=g) * 2).to(torch.bfloat16)
    k, v = ((torch.randn(int(ko[-1]), 2, D, generator=g) * 2).to(torch.bfloat16) for _ in range(2))
    o = G.generalized_dot_product_attention(q.cuda(), k.cuda(), v.cuda(), qo.cuda(), ko.cuda(), max(lq), max(lk), qk_scale=scale,
                                            activation="softmax")
    torch.cuda.synchronize()
    assert G.kernel_status() == 0
    for b in range(len(lq)):
        qb, (kb, vb) = q[qo[b]:qo[b + 1]].double(), (t[ko[b]:ko[b + 1]].double() for t in (k, v))
        p = torch.softmax(torch.einsum("qhd,khd->hqk", qb, kb) * scale, -1)
        assert_close(o[qo[b]:qo[b + 1]], torch.einsum("hqk,khd->qhd", p, vb), f"O[{lq[b]}, {lk[b]}]")


@pytest.mark.parametrize("requests,per,rows,heads", [(1, 5, 9, 1), (3, 64, 32, 2), (2, 700, 60, 2), (40, 33, 200, 2)])
def test_shared_kv_runs_cover_every_row_once(requests, per, rows, heads):
    """Sequences of one KV sequence are scheduled together, in blocks of 128 rows for few rows and 256 for many; a
    sequence longer than the maximum is cut, entries beyond the KV batch are clamped, empty sequences take no rows."""
    rng = np.random.default_rng(per)
    batch = requests * per
    lq = rng.integers(0, rows + 1, batch)
    if rows > 100:
        lq[batch // 2] = rows + 50  # cut at max_q
    index = np.repeat(np.arange(requests), per)
    index[-1] = requests + 3  # clamped to the last request
    index[per // 2] = requests - 1  # breaks a run
    lk = rng.integers(1, 900, requests)
    qo, ko, idx = torch.tensor(np.concatenate([[0], np.cumsum(lq)])).cuda(), torch.tensor(np.concatenate([[0], np.cumsum(lk)])).cuda(), \
        torch.tensor(index).cuda()
    header, items = _schedule(qo, ko, 2, heads, rows, 1000, idx)
    assert header[0] == header[2] == len(items)
    owner = np.full((heads, int(qo[-1])), -1)
    start = qo.cpu().numpy()
    for b, h, first, end in items.tolist():
        assert first < end <= first + 256
        at = owner[h, start[b] + first:start[b] + end]
        assert (at == -1).all() and len(at) == end - first
        at[:] = min(index[b], requests - 1)
    for b in range(batch):
        n = min(lq[b], rows)
        assert (owner[:, start[b]:start[b] + n] == min(index[b], requests - 1)).all()
        assert (owner[:, start[b] + n:start[b + 1]] == -1).all()


@pytest.mark.parametrize("D,act", [(64, "silu"), (128, "gelu_approx"), (128, "softmax")])
@pytest.mark.parametrize("per,rows", [(7, 20), (150, 90)])
def test_shared_kv_runs_give_what_single_sequences_give(G, D, act, per, rows):
    """The same call with a band that reaches every pair is scheduled sequence by sequence.  A row's products, and the order
    of its fp32 sums over the KV tiles, are the same in both: so are the results.  Softmax: single sequences move the reference
    maximum of 32 rows together and runs that of each row, so P is rounded to bf16 (2^-9) from another base; a weighted mean
    of values of a unit then moves by less than that, and by an ulp of bf16, 2^-7 of its value, where it is rounded itself."""
    g = torch.Generator().manual_seed(per)
    rng = np.random.default_rng(per)
    requests, H = 3, 2
    lq, lk = rng.integers(0, rows + 1, requests * per), rng.integers(1, 700, requests)
    qo, ko = (torch.tensor(np.concatenate([[0], np.cumsum(n)])).cuda() for n in (lq, lk))
    q = torch.randn(int(qo[-1]), H, D, generator=g).to(torch.bfloat16).cuda()
    k, v = (torch.randn(int(ko[-1]), H, D, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    index = torch.arange(requests).repeat_interleave(per).cuda()
    out = [G.generalized_dot_product_attention(q, k, v, qo, ko, rows, 700, ad_to_request_offset=index, qk_scale=0.1, activation=act,
                                               window_size=w) for w in (None, 1 << 20)]
    torch.cuda.synchronize()
    assert G.kernel_status() == 0
    if act == "softmax":
        assert_close(out[0], out[1], "runs", atol=2.0 ** -9, rtol=2.0 ** -7)
    else:
        assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("act", ["softmax", "silu", "relu"])
def test_shared_kv_result_does_not_depend_on_the_sequences_beside_it(G, act):
    """Candidates of one request, in one Q tile, with keys that grow: the scores of the second stay within a few units, so that
    alone its softmax keeps the maximum of the first tile, while those of the others (with a factor of 32) move theirs from
    tile to tile.  The rows of the second are the same bits whatever the others hold, infinities and NaN included."""
    g = torch.Generator().manual_seed(5)
    D, lq, kv = 128, [20, 40, 30], 900
    qo, ko = (torch.tensor(np.concatenate([[0], np.cumsum(n)])).cuda() for n in (lq, [kv]))
    q = torch.randn(sum(lq), 2, D, generator=g).to(torch.bfloat16).cuda()
    k, v = (torch.randn(kv, 2, D, generator=g).cuda() for _ in range(2))
    k, v = (k * torch.linspace(0.2, 3.0, kv).cuda().view(-1, 1, 1)).to(torch.bfloat16), v.to(torch.bfloat16)
    rows = []
    for factor in (1.0, 0.0, 32.0, float("inf")):
        x = q.clone()
        x[:20] *= factor
        x[60:] *= -factor
        o = G.generalized_dot_product_attention(x, k, v, qo, ko, 40, kv, ad_to_request_offset=torch.zeros(3, dtype=torch.int64).cuda(),
                                                qk_scale=0.02, activation=act)
        torch.cuda.synchronize()
        assert G.kernel_status() == 0
        rows.append(o[20:60])
    assert rows[0].isfinite().all() and all(torch.equal(rows[0], r) for r in rows[1:])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("long", [0, 9000])
def test_fp8_quantiser_rounds_as_a_division(G, D, long):
    """Both kernels (the one-pass kernel takes batches of 80 rows a sequence and more: those with a long sequence added) against
    the restatement, byte for byte: ragged blocks, more sequences than one round of the owner search holds, zeros, denormals,
    blocks at the 1e-12 scale, infinities and NaN, and every bf16 mantissa over many scales.  A NaN does not count for the scale
    of its block; NaN and, their scale being infinite, infinities become -448."""
    g = torch.Generator().manual_seed(D)
    lens = [130, 0, 1, 128, 127, 384] + [5, 0, 3] * 20 + [128, 128, long]
    off = torch.tensor(np.concatenate([[0], np.cumsum(lens)]))
    T, H = int(off[-1]), 3
    assert (T >= 80 * len(lens)) == (long > 0)
    x = (torch.randn(T, H, D, generator=g) * torch.exp2(torch.randint(-30, 30, (T, H, 1), generator=g).float())).to(torch.bfloat16)
    x[0:131, 0] = 0
    x[131:140, 1] = 1e-39
    x[260:300, 2, 3] = float("inf")
    x[300:310, 2, 5] = -float("inf")
    x[131:200, 2, 7] = float("nan")
    at = int(off[-4])  # two whole tiles
    x[at:at + 128] = 1e-39
    x[at + 128:at + 256] = ((torch.rand(128, H, D, generator=g) * 2 - 1) * 4e-10).to(torch.bfloat16)
    x8, sc, bo = G.quantize_fp8_blockwise(x.cuda(), off.cuda())
    torch.cuda.synchronize()
    r8, rsc, rbo = orc.quantize_fp8_blockwise(x.nan_to_num(0, float("inf"), -float("inf")), off)
    assert torch.equal(bo.cpu(), rbo.to(bo.dtype)) and torch.equal(sc.cpu()[: rsc.shape[0]], rsc)
    want = torch.where(x.isfinite(), r8.view(torch.uint8), torch.full_like(r8, -448.0).view(torch.uint8))
    assert torch.equal(x8.cpu().view(torch.uint8), want)
    assert bool((rsc[int(rbo[-4]):int(rbo[-2])] == 1e-12).all()) and len(want[at + 128:at + 256].unique()) > 100
    n = 1 << 20  # the quotients themselves, scales of every mantissa: one-row sequences, a scale per row
    amax = (torch.randint(0x3F80, 0x4000, (n // 128,), generator=g).to(torch.int16).view(torch.bfloat16)).float()
    v = (torch.rand(n // 128, 128, generator=g) * 2 - 1) * amax[:, None]
    v[:, 0] = amax
    y = v.to(torch.bfloat16).view(-1, 1, 128)
    rows = n // 128
    yo = torch.cat([torch.arange(0, rows + 1), torch.tensor([81 * rows])]) if long else torch.arange(0, rows + 1)
    padded = torch.cat([y, torch.zeros(80 * rows, 1, 128, dtype=y.dtype)]) if long else y
    y8, _, _ = G.quantize_fp8_blockwise(padded.cuda(), yo.cuda())
    scale = (y.float().abs().amax(2, keepdim=True) / 448).clamp_min(1e-12)
    want = (y.float() / scale).clamp(-448, 448).to(torch.float8_e4m3fn)
    assert torch.equal(y8[:rows].cpu().view(torch.uint8), want.view(torch.uint8))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("repeat", [1, 10])
def test_forward_of_items_of_one_to_three_ragged_kv_tiles(D, repeat):
    """The loader asks for all tiles of an item of one or two KV tiles before it zeroes the ragged ones: every combination
    of Q and KV lengths around one and two tiles, against fp64 within the bf16 bound of the kernels.  160 items, at most two
    for each of 148 CTAs; ten times as many take a CTA twice around its ring of work items, from items of three KV tiles
    to those of two and one."""
    import ads_model_kernel_library_b200.gdpa as G

    g = torch.Generator().manual_seed(D)
    edges = [1, 127, 128, 129, 255, 256, 257, 300]
    lq, lk = [a for a in edges for _ in edges] * repeat, [b for _ in edges for b in edges] * repeat
    qo, ko = (torch.tensor(np.concatenate([[0], np.cumsum(n)])) for n in (lq, lk))
    q = torch.randn(int(qo[-1]), 2, D, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(int(ko[-1]), 2, D, generator=g).to(torch.bfloat16) for _ in range(2))
    o = G.generalized_dot_product_attention(q.cuda(), k.cuda(), v.cuda(), qo.cuda(), ko.cuda(), 300, 300, qk_scale=1 / 64,
                                            activation="gelu_approx")
    torch.cuda.synchronize()
    assert G.kernel_status() == 0
    for b in range(len(lq)):
        qb, (kb, vb) = q[qo[b]:qo[b + 1]].double(), (t[ko[b]:ko[b + 1]].double() for t in (k, v))
        p = torch.nn.functional.gelu(torch.einsum("qhd,khd->hqk", qb, kb), approximate="tanh") / 64
        assert_close(o[qo[b]:qo[b + 1]], torch.einsum("hqk,khd->qhd", p, vb), f"O[{lq[b]}, {lk[b]}]")


@pytest.mark.parametrize("scale,value", [("0x1.2da85cp-1", 0.0), ("0x1.2da864p-1", 0.0), ("0x1.2da850p-1", 2.0 ** -9)])
def test_fp8_softmax_rounds_the_exponent_before_the_factor_of_p(G, scale, value):
    """P is stored as e4m3(2^7 exp2(x)), x = c S - m rounded to fp32.  The midpoint between 0 and the smallest e4m3, 2^-10,
    is x = -17.  One key has S = 0 (m = 0, P = 2^7, its V row is 0), 127 have S = -20 and V = 1, so a row is
    127 e4m3(2^7 exp2(x)) over the row sum.  With the first scale c S is 0.75 * 2^-20 above -17, which fp32 rounds to -17
    (spacing 2^-19) and the conversion to 0; as a term of the exponent 2^7 would move the sum to -10, where the spacing is
    2^-20, and P to 2^-9.  The second scale gives c S below -17, the third 5.4 * 2^-19 above."""
    D = 128
    q, k, v = (torch.zeros(128, 1, D) for _ in range(3))
    q[:, 0, 0] = 1.0
    k[1:, 0, 0] = -20.0
    v[1:] = 1.0
    off, blocks, one = torch.tensor([0, 128]).cuda(), torch.tensor([0, 1]).cuda(), torch.ones(1, 1).cuda()
    o = G.generalized_dot_product_attention_fp8(*(t.to(torch.float8_e4m3fn).cuda() for t in (q, k, v)), one, one, one, blocks, blocks,
                                                off, off, 128, 128, qk_scale=float.fromhex(scale))
    torch.cuda.synchronize()
    assert G.kernel_status() == 0
    want = torch.tensor(127 * value / 128 / (1 + 127 * 2.0 ** -17)).to(torch.bfloat16)
    assert torch.equal(o.cpu(), want.expand(o.shape))


@pytest.mark.parametrize("act", ["softmax", "gelu_approx"])
def test_fp8_forward_with_empty_kv_sequences_and_scales_of_exactly_the_blocks(G, act):
    """A sequence without keys has no row in the scales: behind the last block there is nothing to read.  Its output rows
    are zero; the other rows are those of the same call with the rows that the quantiser allocates behind the blocks."""
    lq, lk = [130, 0, 300, 7, 40], [0, 64, 300, 0, 0]
    g = torch.Generator().manual_seed(3)
    qo, ko = (torch.tensor(np.concatenate([[0], np.cumsum(n)])).cuda() for n in (lq, lk))
    q, k, v = (torch.randn(n, 2, 128, generator=g).to(torch.bfloat16).cuda() for n in (sum(lq), sum(lk), sum(lk)))
    (q8, sq, qb), (k8, sk, kb), (v8, sv, _) = (G.quantize_fp8_blockwise(t, o) for t, o in ((q, qo), (k, ko), (v, ko)))
    out = []
    for rows in (len(sk), int(kb[-1])):
        out.append(G.generalized_dot_product_attention_fp8(q8, k8, v8, sq, sk[:rows].clone(), sv[:rows].clone(), qb, kb, qo, ko, 300, 300,
                                                           qk_scale=0.1, activation=act))
        torch.cuda.synchronize()
        assert G.kernel_status() == 0
    assert torch.equal(out[0], out[1])
    empty = torch.cat([out[1][:130], out[1][430:]])
    assert bool((empty == 0).all()) and bool(out[1][130:430].isfinite().all()) and bool((out[1][130:430] != 0).any())


@pytest.mark.parametrize("call,mode", [("fp8", 2), ("fp8", 1), ("window", 2), ("no index", 2), ("no index", 1), ("backward", 0),
                                       ("backward", 2)])
def test_a_kernel_refuses_a_schedule_it_cannot_walk(G, monkeypatch, call, mode):
    """Items of another mode name other rows and blocks: the kernel walks none of them, writes the mode it found to the
    status word, and the next call raises it."""
    from ads_model_kernel_library_b200.gdpa import _cabi, ops

    D, lens = 128, [300, 5, 700]
    off = torch.tensor(np.concatenate([[0], np.cumsum(lens)])).cuda()
    index = torch.arange(len(lens)).cuda()
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(sum(lens), 2, D, generator=g).to(torch.bfloat16).cuda().requires_grad_(call == "backward") for _ in range(3))
    build = ops._build_schedule

    def other_mode(wanted, qo, ko, batch, heads, rows, max_q, max_kv, kv_index=None, start_end=False):
        wrong = (wanted == _cabi.GDPA_SCHED_BWD) if call == "backward" else True
        return build(mode if wrong else wanted, qo, ko, batch, heads, rows, max_q, max_kv, index if wrong and mode == 2 else kv_index)

    monkeypatch.setattr(ops, "_build_schedule", other_mode)
    if call == "fp8":
        (q8, sq, b), (k8, sk, _), (v8, sv, _) = (G.quantize_fp8_blockwise(t, off) for t in (q, k, v))
        G.generalized_dot_product_attention_fp8(q8, k8, v8, sq, sk, sv, b, b, off, off, 700, 700)
    elif call == "window":
        G.generalized_dot_product_attention(q, k, v, off, off, 700, 700, ad_to_request_offset=index, window_size=64)
    else:
        o = G.generalized_dot_product_attention(q, k, v, off, off, 700, 700, activation="relu")
        if call == "backward":
            o.sum().backward()
    torch.cuda.synchronize()
    monkeypatch.undo()
    with pytest.raises(RuntimeError, match=f"schedule of mode {mode}"):
        G.generalized_dot_product_attention(q, k, v, off, off, 700, 700, activation="relu")
    G.generalized_dot_product_attention(q, k, v, off, off, 700, 700, activation="relu")
    assert G.kernel_status() == 0
