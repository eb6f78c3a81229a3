"""The tcgen05 ranking / top-k kernel and the evaluator path built on it, against fp32 PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

from dice_embeddings_b200.ops import kernels as K
from dice_embeddings_b200.ops.eval_rank import FusedRanker

DEV = torch.device("cuda:0")


def _operands(nx, ny, D, seed):
    torch.manual_seed(seed)
    x = (torch.randn(nx, D, device=DEV) * 0.3).to(torch.bfloat16)
    y = (torch.randn(ny, D, device=DEV) * 0.3).to(torch.bfloat16)
    return x, y


def _random_filter(nx, ny, per_row, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    counts = torch.randint(0, per_row + 1, (nx,), generator=g)
    ptr = torch.zeros(nx + 1, dtype=torch.int64)
    ptr[1:] = torch.cumsum(counts, 0)
    cols = torch.randint(0, ny, (int(ptr[-1]),), generator=g, dtype=torch.int32)
    return ptr.to(DEV), cols.to(DEV)


def _ref_ranks(scores, tgt_idx, tgt_score, ptr, cols):
    nx = scores.shape[0]
    ar = torch.arange(nx, device=DEV)
    beats = scores > tgt_score[:, None]
    beats[ar, tgt_idx.long()] = False
    greater = beats.sum(1)
    rows = torch.repeat_interleave(ar, ptr[1:] - ptr[:-1])
    mask = torch.zeros_like(beats)
    mask[rows, cols.long()] = True          # duplicates in the filter list count once here ...
    mask[ar, tgt_idx.long()] = False
    filt_unique = (beats & mask).sum(1)
    return greater, filt_unique


@pytest.mark.parametrize("nx,ny,D", [(128, 128, 64), (300, 5000, 128), (257, 1300, 256), (1000, 20000, 256)])
def test_eval_rank_counts_and_filter(nx, ny, D):
    x, y = _operands(nx, ny, D, nx + ny)
    tgt = torch.randint(0, ny, (nx,), device=DEV, dtype=torch.int32)
    ptr, cols = _random_filter(nx, ny, 6, 1)
    # the CSR of a knowledge graph has no duplicates inside a row: make the rows unique
    key = torch.repeat_interleave(torch.arange(nx, device=DEV), ptr[1:] - ptr[:-1]) * ny + cols.long()
    key = torch.unique(key)
    rows_u, cols = key // ny, (key % ny).to(torch.int32)
    ptr = torch.zeros(nx + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(rows_u, minlength=nx), 0)
    r = FusedRanker(y)
    ranks = r.ranks(x, tgt, ptr, cols)
    scores = x.float() @ y.float().t()
    tgt_score = scores[torch.arange(nx, device=DEV), tgt.long()]
    greater, filt = _ref_ranks(scores, tgt, tgt_score, ptr, cols)
    ref = 1 + greater - filt
    diff = (ranks - ref).abs()
    assert diff.max() <= 2, diff.max()          # only scores within rounding of the target may flip
    assert (diff > 0).float().mean() < 0.02


def test_eval_sparse_target_scores():
    x, y = _operands(500, 3000, 256, 3)
    tgt = torch.randint(0, 3000, (500,), device=DEV, dtype=torch.int32)
    out = torch.zeros(500, device=DEV)
    K.eval_sparse(x, y, tgt, out, None)
    ref = (x.float() * y.float()[tgt.long()]).sum(1)
    assert torch.allclose(out, ref, atol=1e-3, rtol=1e-3)


@pytest.mark.parametrize("nx,ny,D,k", [(5, 4000, 64, 10), (200, 30000, 128, 10), (130, 3000, 256, 32), (1, 100000, 256, 3)])
def test_eval_topk(nx, ny, D, k):
    x, y = _operands(nx, ny, D, k + nx)
    r = FusedRanker(y)
    sc, ix = r.topk(x, k)
    ref_s, ref_i = torch.topk(x.float() @ y.float().t(), k, dim=1)
    assert torch.allclose(sc, ref_s, atol=2e-3, rtol=1e-3)
    same = (ix == ref_i).float().mean()
    assert same > 0.97, same                     # swaps only between entities whose scores tie within rounding
    assert (torch.sort(sc, dim=1, descending=True).values == sc).all()


def test_eval_rank_bias_and_cyclic_shards_add_up():
    """Two cyclic row shards with a per-entity bias give the same counts and top-k as the whole table."""
    nx, ny, D = 300, 7001, 128
    x, y = _operands(nx, ny, D, 11)
    bias = torch.randn(ny, device=DEV) * 0.5
    tgt = torch.randint(0, ny, (nx,), device=DEV, dtype=torch.int32)
    scores = x.float() @ y.float().t() + bias
    tgt_score = scores[torch.arange(nx, device=DEV), tgt.long()].contiguous()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    greater = torch.zeros(nx, dtype=torch.int32, device=DEV)
    cands = []
    for rank in range(2):
        ys, bs = y[rank::2].contiguous(), bias[rank::2].contiguous()
        cap = K.eval_rank_cand_cap(nx, ys.shape[0], D, 5)
        cs = torch.full((nx, cap), float("-inf"), device=DEV)
        ci = torch.full((nx, cap), -1, dtype=torch.int32, device=DEV)
        cc = torch.zeros(nx, dtype=torch.int32, device=DEV)
        K.eval_rank(x, ys, tgt_score, tgt, greater, status, col_bias=bs, y_offset=rank, y_stride=2, k=5,
                    cand_score=cs, cand_idx=ci, cand_count=cc)
        cands.append((cs, ci))
    torch.cuda.synchronize()
    K.check_status(status)
    beats = scores > tgt_score[:, None]
    beats[torch.arange(nx, device=DEV), tgt.long()] = False
    diff = (greater.long() - beats.sum(1)).abs()
    assert diff.max() <= 2 and (diff > 0).float().mean() < 0.02
    cs = torch.cat([c[0] for c in cands], 1)
    ci = torch.cat([c[1] for c in cands], 1)
    top_s, pos = torch.topk(cs, 5, dim=1)
    top_i = torch.gather(ci, 1, pos).long()
    ref_s, ref_i = torch.topk(scores, 5, dim=1)
    assert torch.allclose(top_s, ref_s, atol=2e-3, rtol=1e-3)
    assert (top_i == ref_i).float().mean() > 0.97


def test_evaluator_fused_path_agrees_with_torch_path(tmp_path):
    from dice_embeddings_b200.data.synthetic import zipf_kg
    from dice_embeddings_b200.data.vocab import er_csr
    from dice_embeddings_b200.evaluation.ranking import metrics_from_ranks, tail_ranks
    from dice_embeddings_b200.models import initialize_model
    triples = zipf_kg(2000, 20, 30000, seed=5)
    model, _ = initialize_model({"model": "ComplEx", "embedding_dim": 96, "num_entities": 2000, "num_relations": 20,
                                 "scoring_technique": "KvsAll"})
    model = model.to(DEV).eval()
    csr = er_csr(triples, 20)
    test = torch.as_tensor(triples[:3000])
    slow = tail_ranks(model, test, csr, 1024, fused=False)
    fast = tail_ranks(model, test, csr, 1024, fused=True)
    # the evaluator's fused path re-scores the undecided band in fp32: same ranks as the fp32 path
    assert (slow == fast).float().mean() > 0.999 and (slow - fast).abs().max() <= 1
    a, b = metrics_from_ranks(slow), metrics_from_ranks(fast)
    assert abs(a["MRR"] - b["MRR"]) < 1e-5


@pytest.mark.parametrize("nx,ny,D", [(300, 5000, 128), (1000, 20000, 256), (64, 3000, 96)])
def test_exact_mode_reproduces_fp32_ranks(nx, ny, D):
    """fp32 operands that are *not* bf16-representable: the band re-scoring must undo the rounding of the GEMM."""
    torch.manual_seed(nx)
    x = torch.randn(nx, D, device=DEV) * 0.3
    y = torch.randn(ny, D, device=DEV) * 0.3
    tgt = torch.randint(0, ny, (nx,), device=DEV, dtype=torch.int32)
    ptr, cols = _random_filter(nx, ny, 5, 2)
    key = torch.unique(torch.repeat_interleave(torch.arange(nx, device=DEV), ptr[1:] - ptr[:-1]) * ny + cols.long())
    rows_u, cols = key // ny, (key % ny).to(torch.int32)
    ptr = torch.zeros(nx + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(rows_u, minlength=nx), 0)
    scores = x.double() @ y.double().t()                     # oracle in fp64
    tgt_score = scores[torch.arange(nx, device=DEV), tgt.long()]
    greater, filt = _ref_ranks(scores, tgt, tgt_score, ptr, cols)
    ref = 1 + greater - filt
    exact = FusedRanker(y, exact=True).ranks(x, tgt, ptr, cols)
    rough = FusedRanker(y, exact=False).ranks(x, tgt, ptr, cols)
    assert (exact == ref).float().mean() > 0.998 and (exact - ref).abs().max() <= 1   # fp32 vs fp64 ties only
    assert (rough == ref).float().mean() < (exact == ref).float().mean()            # the band pass is what fixes them


@pytest.mark.parametrize("adversarial", [False, True])
def test_two_stage_topk_over_a_large_table(adversarial):
    """Tables above the two-stage limit: threshold from a strided sample of the rows, then one collecting pass; the
    sample stays representative when the rows are sorted by norm, and nothing in the call waits for the GPU."""
    nx, ny, D, k = 70, 300000, 128, 10
    x, y = _operands(nx, ny, D, 9)
    if adversarial:
        scale = torch.linspace(0.05, 3.0, ny, device=DEV)[:, None]
        y = (y.float() * scale).to(torch.bfloat16)
    r = FusedRanker(y)
    assert ny > r.TWO_STAGE_ROWS
    sc, ix = r.topk(x, k)
    ref_s, ref_i = torch.topk(x.float() @ y.float().t(), k, dim=1)
    assert torch.allclose(sc, ref_s, atol=5e-3, rtol=2e-3)
    assert (ix == ref_i).float().mean() > 0.97


@pytest.mark.parametrize("nx,ny,D", [(1, 1, 64), (129, 127, 64), (256, 128, 128), (257, 129, 128), (600, 40000, 256), (100, 300, 256)])
@pytest.mark.parametrize("bias", [False, True])
def test_masked_counts(nx, ny, D, bias):
    """Columns in the mask never count; one and two row planes, partial planes and tiles.  Integer operands: exact sums."""
    torch.manual_seed(nx + ny)
    x = torch.randint(-3, 4, (nx, D), device=DEV).to(torch.bfloat16)
    y = torch.randint(-3, 4, (ny, D), device=DEV).to(torch.bfloat16)
    b = torch.randint(-9, 10, (ny,), device=DEV).float() if bias else None
    scores = x.float() @ y.float().t() + (b if bias else 0.0)
    tgt = torch.randint(0, ny, (nx,), device=DEV, dtype=torch.int32)
    ts = scores[torch.arange(nx, device=DEV), tgt.long()].contiguous()
    drop = torch.rand(nx, ny, device=DEV) < 0.3
    words = (ny + 127) // 128 * 4
    mask = torch.zeros(nx, words, dtype=torch.int32, device=DEV)
    ptr = torch.zeros(nx + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = drop.sum(1).cumsum(0)
    K.filter_mask(mask, ny, ptr=ptr, cols=drop.nonzero()[:, 1].to(torch.int32).contiguous())
    greater = torch.zeros(nx, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    K.rank_count(x, y, ts, tgt, greater, status, col_bias=b, mask=mask)
    assert int(status) == 0
    beats = (scores > ts[:, None]) & ~drop
    assert torch.equal(greater.long(), beats.sum(1))


@pytest.mark.parametrize("pairs", [1, 31, 33, 34, 1100, 40000])
def test_filter_mask_by_pair(pairs):
    """The pair search over sorted keys finds exactly the stored pairs (32-ary search: sizes around its step)."""
    g = torch.Generator().manual_seed(pairs)
    num_b, ny = 7, 333
    keys = torch.randperm(3 * pairs, generator=g)[:pairs].sort().values
    counts = torch.randint(0, 5, (pairs,), generator=g)
    offsets = torch.zeros(pairs + 1, dtype=torch.int64)
    offsets[1:] = counts.cumsum(0)
    values = torch.randint(0, ny, (int(offsets[-1]) + 1,), generator=g)
    ask = torch.cat([torch.arange(0, 40), torch.randint(0, 3 * pairs + 5, (500,), generator=g), torch.tensor([3 * pairs - 1, 3 * pairs])])
    ab = torch.stack((ask // num_b, ask % num_b, torch.zeros_like(ask)), 1).to(DEV)
    mask = torch.zeros(len(ask), 12, dtype=torch.int32, device=DEV)
    K.filter_mask(mask, ny, ab=ab, num_b=num_b, keys=keys.to(DEV), offsets=offsets.to(DEV), values=values.to(DEV))
    where = {int(k): i for i, k in enumerate(keys)}
    got = mask.cpu()
    for row, k in enumerate(ask.tolist()):
        want = torch.zeros(12 * 32, dtype=torch.bool)
        if k in where:
            want[values[offsets[where[k]]:offsets[where[k] + 1]]] = True
        bits = (got[row].view(-1, 1) >> torch.arange(32)) & 1
        assert torch.equal(bits.bool().reshape(-1), want), k


def _check_topk(sc, ix, scores, k):
    ref, _ = torch.topk(scores, k, dim=1)
    assert torch.equal(sc, ref)
    assert torch.equal(torch.gather(scores, 1, ix), sc) and all(len(set(r)) == k for r in ix.tolist())


@pytest.mark.parametrize("n", [1, 2, 33, 128, 129, 2047, 40000, 140000])
@pytest.mark.parametrize("B,D", [(1, 64), (4, 128), (5, 64), (130, 128), (300, 256)])
def test_topk_integer_scores_with_ties(n, B, D):
    """Small integers make exact sums and many ties: best scores, distinct ids that have them; few queries (one scan) and
    many (tensor cores), fewer columns than groups, one tile, several, the two-stage path; a constant table."""
    torch.manual_seed(n + B)
    x = torch.randint(-1, 2, (B, D), device=DEV).to(torch.bfloat16)
    y = torch.randint(-1, 2, (n, D), device=DEV).to(torch.bfloat16)
    if n > 131072:   # few values on the sample's floor: otherwise the ties alone would not fit any list
        y = (y.float() + torch.randint(-3, 4, (n, D), device=DEV)).to(torch.bfloat16)
    for k in sorted({1, min(n, 10), min(n, 32)}):
        r = FusedRanker(y)
        sc, ix = r.topk(x.float() if B == 1 else x, k)
        r.check()
        _check_topk(sc, ix, x.float() @ y.float().t(), k)
    if n <= 40000:
        bias = torch.randint(-2, 3, (n,), device=DEV).float()
        r = FusedRanker(torch.zeros_like(y), col_bias=bias)       # n columns, five different scores
        sc, ix = r.topk(x, min(n, 32))
        r.check()
        _check_topk(sc, ix, bias.expand(B, -1), min(n, 32))


def test_topk_skips_what_is_not_a_score():
    x = torch.ones(3, 64, device=DEV)
    y = torch.arange(200, device=DEV).float()[:, None].expand(-1, 64).contiguous()
    bias = torch.zeros(200, device=DEV)
    bias[150:] = float("-inf")
    bias[140:150] = float("nan")
    for q in (x, x.repeat(3, 1)):
        r = FusedRanker(y[:, :64], col_bias=bias)
        sc, ix = r.topk(q, 5)
        assert ix.tolist() == [[139, 138, 137, 136, 135]] * q.shape[0] and torch.isfinite(sc).all()
        r = FusedRanker(y[148:], col_bias=bias[148:].contiguous())
        sc, ix = r.topk(q, 5)
        assert (ix == -1).all() and (sc == float("-inf")).all()


def test_split_scores_stay_within_the_margin():
    """The margin of the band must cover the error of the split GEMM: no pair outside the band may be decided wrongly."""
    for D in (64, 128, 256):
        torch.manual_seed(D)
        x, y = torch.randn(400, D, device=DEV), torch.randn(6000, D, device=DEV) * torch.rand(6000, 1, device=DEV)
        exact = x.double() @ y.double().t()
        tgt = torch.randint(0, 6000, (400,), device=DEV, dtype=torch.int32)
        ts = exact[torch.arange(400, device=DEV), tgt.long()].float().contiguous()
        factor = float(y.norm(dim=1).max()) * FusedRanker.MARGIN[D]
        xh, xl, _, margin = K.split_rows(x, D, margin_factor=factor)
        yh, yl, _, _ = K.split_rows(y, D)
        greater = torch.zeros(400, dtype=torch.int32, device=DEV)
        rows, cols = (torch.empty(1 << 20, dtype=torch.int32, device=DEV) for _ in range(2))
        count = torch.zeros(1, dtype=torch.int64, device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        K.rank_count(xh, yh, ts, tgt, greater, status, x_lo=xl, y_lo=yl, margin=margin, band_rows=rows, band_cols=cols,
                     band_count=count)
        n = int(count)
        assert int(status) == 0 and n < 0.01 * 400 * 6000
        band = torch.zeros(400, 6000, dtype=torch.bool, device=DEV)
        band[rows[:n].long(), cols[:n].long()] = True
        beats = exact > ts[:, None].double()
        beats[torch.arange(400, device=DEV), tgt.long()] = False
        assert torch.equal(greater.long(), (beats & ~band).sum(1))


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("cap", [1, 45, 1000])
def test_full_band_list_has_no_gaps(split, cap):
    """A list that runs full is reported and holds a listed pair in every slot: the second pass reads all of them.  Margins
    of infinity put every pair but the targets' own into the band."""
    nx, ny, D = 70, 500, 64
    x, y = _operands(nx, ny, D, cap)
    lo = dict(x_lo=torch.zeros_like(x), y_lo=torch.zeros_like(y)) if split else {}
    tgt = torch.randint(0, ny, (nx,), device=DEV, dtype=torch.int32)
    rows, cols = (torch.full((cap,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    count = torch.zeros(1, dtype=torch.int64, device=DEV)
    greater, status = torch.zeros(nx, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    K.rank_count(x, y, torch.zeros(nx, device=DEV), tgt, greater, status, margin=torch.full((nx,), float("inf"), device=DEV),
                 band_rows=rows, band_cols=cols, band_count=count, **lo)
    assert int(status) != 0 and int(count) == nx * (ny - 1) and int(greater.sum()) == 0
    r, c = rows.long(), cols.long()
    assert ((r >= 0) & (r < nx) & (c >= 0) & (c < ny)).all() and (c != tgt.long()[r.clamp_min(0)]).all()
    assert torch.unique(r * ny + c).numel() == cap


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("masked", [False, True])
def test_repeated_answers_in_a_filter(exact, masked):
    """An answer that a list names several times is subtracted as often as it is named, whether the answers are masked or
    scored one by one; lists without repeats, with the target, and empty ones.  Integer operands: exact scores."""
    from dice_embeddings_b200.evaluation.ranking import filtered_rank_from_scores
    torch.manual_seed(5)
    nx, ny, D = 60, 400, 64
    x, y = torch.randint(-3, 4, (nx, D), device=DEV).float(), torch.randint(-3, 4, (ny, D), device=DEV).float()
    tgt = torch.randint(0, ny, (nx,), device=DEV)
    lists = [torch.randint(0, 25, (90,)) if i % 3 == 0 else torch.randperm(ny)[:40] if i % 3 == 1 else torch.zeros(0).long() for i in range(nx)]
    lists[0][7:9] = int(tgt[0])
    lists[1] = torch.arange(129) // 2 * 3           # more than one round of the mask kernel, repeats across its words
    ptr = torch.zeros(nx + 1, dtype=torch.int64)
    ptr[1:] = torch.tensor([len(a) for a in lists]).cumsum(0)
    rows, cols = torch.repeat_interleave(torch.arange(nx), ptr[1:] - ptr[:-1]).to(DEV), torch.cat(lists).to(DEV)
    r = FusedRanker(y, exact=exact)
    r._mask_pays = lambda *a: masked
    got = r.ranks(x, tgt, ptr.to(DEV), cols.to(torch.int32))
    r.check()
    assert torch.equal(got, filtered_rank_from_scores(x @ y.t(), tgt, rows, cols))


def test_a_target_of_minus_zero():
    """-0 is not below +0: scores of zero are not above a target of -0, in the counting and in the band form."""
    x, y = torch.zeros(5, 64, dtype=torch.bfloat16, device=DEV), _operands(1, 300, 64, 0)[1]
    bias = torch.zeros(300, device=DEV)
    bias[7], bias[9] = 1e-38, -0.0
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for band in (False, True):
        kw = {}
        if band:
            lists = [torch.zeros(2000, dtype=torch.int32, device=DEV) for _ in range(2)]
            count = torch.zeros(1, dtype=torch.int64, device=DEV)
            kw = dict(margin=torch.zeros(5, device=DEV), band_rows=lists[0], band_cols=lists[1], band_count=count)
        greater = torch.zeros(5, dtype=torch.int32, device=DEV)
        K.rank_count(x, y, torch.full((5,), -0.0, device=DEV), None, greater, status, col_bias=bias, **kw)
        assert greater.tolist() == [1] * 5 and int(status) == 0 and (not band or int(count) == 0)


@pytest.mark.parametrize("D", [64, 256])
@pytest.mark.parametrize("size", [1e-2, 30.0, 1000.0])
def test_exact_ranks_with_a_bias_far_above_the_scores(D, size):
    """A bias that rounds most of the score away leaves few different sums; the ranks are still those of the fp32 sums, which
    the gather-dots give with the same order of additions as the second pass."""
    torch.manual_seed(0)
    n, B = 3000, 300
    x, y = torch.randn(B, D, device=DEV) * 1e-4, torch.randn(n, D, device=DEV)
    bias = torch.full((n,), size, device=DEV)
    bias[::7] = float("-inf")
    tgt = 1 + 7 * torch.randint(0, n // 7, (B,), device=DEV, dtype=torch.int32)
    r = FusedRanker(y, col_bias=bias, exact=True)
    got = r.ranks(x, tgt)
    r.check()
    ts, above = torch.zeros(B, device=DEV), torch.zeros(B, dtype=torch.int32, device=DEV)
    K.eval_sparse(x, y, tgt, ts, above, torch.arange(B + 1, device=DEV) * n, torch.arange(n, device=DEV, dtype=torch.int32).repeat(B),
                  col_bias=bias)
    assert torch.equal(got, 1 + above.long())


def _best(x, y, k):
    return torch.cat([torch.topk(x[i:i + 256].float() @ y.float().t(), k, dim=1).values for i in range(0, x.shape[0], 256)])


def test_two_stage_lists_hold_what_beats_the_sample():
    """The best of a sample of one row in 61 is beaten by 61 rows on average and by ten times as many once in 20 000 queries:
    16 384 queries for their single best row, and the capacity against the tail of the distribution for every k."""
    torch.manual_seed(0)
    y = torch.randn(2_000_000, 64, device=DEV).to(torch.bfloat16)
    r = FusedRanker(y)
    for _ in range(2):
        x = torch.randn(8192, 64, device=DEV).to(torch.bfloat16)
        sc, ix = r.topk(x, 1)
        assert int(r.overflow) == 0
        assert torch.allclose(sc, _best(x, y, 1), atol=1e-3)
    for k in range(1, 33):       # P(gamma of order k > c) = sum over j < k of c^j e^-c / j!
        c = torch.tensor(r._list_capacity(k) / (y.shape[0] / r.SAMPLE_ROWS), dtype=torch.float64)
        j = torch.arange(k, dtype=torch.float64)
        assert float(torch.exp(j * c.log() - c - torch.lgamma(j + 1)).sum()) < 6.1e-13, k


@pytest.mark.parametrize("order", ["end", "periodic"])
def test_two_stage_sample_covers_the_table(order):
    """Rows ten times as long as the rest, where a sample of every (n // S)-th row has none: at the end, and at one place of
    its period."""
    n, k = 160000, 10
    x, y = _operands(70, n, 64, 3)
    y = y.float()
    if order == "end":
        y[131072:] *= 10
    else:
        y[3::4] *= 10
    y = y.to(torch.bfloat16)
    r = FusedRanker(y)
    sc, ix = r.topk(x, k)
    r.check()
    assert torch.allclose(sc, _best(x, y, k), atol=1e-2, rtol=1e-3)
    rows = r._sample_rows()
    assert rows.shape == (r.SAMPLE_ROWS,) and (rows[1:] > rows[:-1]).all() and int(rows[0]) < 8 and int(rows[-1]) >= n - 8


def test_a_full_list_is_reported_and_the_next_call_is_right():
    n, k = 140000, 3
    x, y = _operands(40, n, 64, 4)
    r = FusedRanker(y)
    r._list_capacity = lambda kk: 2
    r.topk(x, k)
    with pytest.raises(K.KernelError):
        r.check()
    r.GROUP_MAX_BYTES = 16 * ((n + 127) // 128) * 7        # seven queries per pass
    sc, ix = r.topk(x, k)
    r.check()
    _check_topk_close(sc, ix, x, y, k)


def _check_topk_close(sc, ix, x, y, k):
    scores = x.float() @ y.float().t()
    assert torch.allclose(sc, torch.topk(scores, k, dim=1).values, atol=1e-3)
    assert torch.allclose(torch.gather(scores, 1, ix), sc, atol=1e-3)


def test_collecting_with_counts_and_a_band_without():
    """``eval_rank`` counts beside collecting when it is given a target and a count buffer, and lists a band without one."""
    nx, ny, D = 150, 2000, 64
    x, y = _operands(nx, ny, D, 21)
    scores = x.float() @ y.float().t()
    tgt = torch.randint(0, ny, (nx,), device=DEV, dtype=torch.int32)
    ts = scores[torch.arange(nx, device=DEV), tgt.long()].contiguous()
    want = torch.zeros(nx, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    K.eval_rank(x, y, ts, tgt, want, status)
    greater, count = torch.zeros(nx, dtype=torch.int32, device=DEV), torch.zeros(nx, dtype=torch.int32, device=DEV)
    lists = torch.full((nx, 100), float("-inf"), device=DEV), torch.full((nx, 100), -1, dtype=torch.int32, device=DEV)
    floor = torch.topk(scores, 20, dim=1).values[:, -1].contiguous() - 1e-3
    K.eval_rank(x, y, ts, tgt, greater, status, k=-1, cand_score=lists[0], cand_idx=lists[1], cand_count=count, row_floor=floor)
    assert torch.equal(greater, want) and int(want.sum()) > 0 and ((count >= 20) & (count < 25)).all()
    rows, cols = (torch.zeros(nx * ny, dtype=torch.int32, device=DEV) for _ in range(2))
    n = torch.zeros(2, dtype=torch.int64, device=DEV)
    for i, g in enumerate((torch.zeros(nx, dtype=torch.int32, device=DEV), None)):
        K.eval_rank(x, y, ts, tgt, g, status, margin=torch.full((nx,), 0.05, device=DEV), band_rows=rows, band_cols=cols,
                    band_count=n[i:i + 1])
    assert int(status) == 0 and int(n[0]) > 0 and int(n[0]) == int(n[1])
