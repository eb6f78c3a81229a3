"""Device sampling kernels and the fused sampled-candidate training step against PyTorch autograd."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

from dice_embeddings_b200.data.datasets import OnevsSample, TriplePredictionDataset
from dice_embeddings_b200.data.synthetic import zipf_kg
from dice_embeddings_b200.models import initialize_model
from dice_embeddings_b200.ops import kernels as K
from dice_embeddings_b200.ops import sampling
from dice_embeddings_b200.ops.sampled_step import FusedSampledEngine

DEV = torch.device("cuda:0")


def test_uniform_int_range_reproducibility_and_spread():
    a = sampling.uniform_int(1000, (200001,), DEV, seed=7)
    b = sampling.uniform_int(1000, (200001,), DEV, seed=7)
    c = sampling.uniform_int(1000, (200001,), DEV, seed=8)
    assert a.min() >= 0 and a.max() < 1000 and torch.equal(a, b) and not torch.equal(a, c)
    counts = torch.bincount(a, minlength=1000).float()
    assert counts.min() > 120 and counts.max() < 290          # expectation 200, sd 14
    big = sampling.uniform_int(10 ** 12, (1000,), DEV, seed=1)
    assert big.max() > 10 ** 10 and big.max() < 10 ** 12


@pytest.mark.parametrize("per_negative", [False, True])
def test_neg_sample_layout_and_semantics(per_negative):
    B, k, NE = 500, 4, 3000
    pos = torch.stack((torch.randint(0, NE, (B,)), torch.randint(0, 9, (B,)), torch.randint(0, NE, (B,))), 1).to(DEV)
    x = torch.zeros(B * (1 + k), 3, dtype=torch.int64, device=DEV)
    y = torch.zeros(B * (1 + k), device=DEV)
    h, r, t = (torch.zeros(B * (1 + k), dtype=torch.int64, device=DEV) for _ in range(3))
    step = torch.tensor([3], device=DEV)
    K.neg_sample(pos, k, NE, 11, 0, y, x=x, hrt=(h, r, t), label_pos=0.9, label_neg=0.1,
                 per_negative_coin=per_negative, step=step)
    assert torch.equal(x[:B], pos) and torch.equal(torch.stack((h, r, t), 1), x)
    assert torch.allclose(y[:B], torch.full((B,), 0.9, device=DEV)) and torch.allclose(y[B:], torch.full((B * k,), 0.1, device=DEV))
    neg = x[B:].reshape(k, B, 3)
    assert (neg[:, :, 1] == pos[:, 1]).all()
    head_changed = neg[:, :, 0] != pos[:, 0]
    tail_changed = neg[:, :, 2] != pos[:, 2]
    assert not (head_changed & tail_changed).any()
    if per_negative:
        assert 0.3 < head_changed.float().mean() < 0.7
    else:
        assert head_changed.float().mean() > 0.95 or tail_changed.float().mean() > 0.95
    assert x.min() >= 0 and x[:, [0, 2]].max() < NE
    # same (seed, offset + step) -> same draw; another step -> another draw
    x2 = torch.zeros_like(x)
    K.neg_sample(pos, k, NE, 11, 3, y, x=x2, per_negative_coin=per_negative)
    assert torch.equal(x, x2)
    K.neg_sample(pos, k, NE, 11, 4, y, x=x2, per_negative_coin=per_negative)
    assert not torch.equal(x, x2)


def _pair(name, D, NE=600, NR=12, scoring="NegSample"):
    torch.manual_seed(1)
    args = dict(model=name, embedding_dim=D, num_entities=NE, num_relations=NR, optim="SGD", learning_rate=1.0,
                scoring_technique=scoring, p=0, q=1)
    m1, _ = initialize_model(dict(args))
    m2, _ = initialize_model(dict(args))
    m2.load_state_dict(m1.state_dict())
    for m in (m1, m2):
        m.to(DEV)
        if name == "Keci":
            with torch.no_grad():
                m.q_coefficients.weight.fill_(0.5)
    return m1, m2


def _compare_updates(ref, fused, lr):
    for (n, p_ref), (_, p) in zip(ref.named_parameters(), fused.named_parameters()):
        if p_ref.grad is None:
            continue
        start = p_ref.detach() + lr * p_ref.grad
        d_ref, d = p_ref.detach() - start, p.detach() - start
        scale = d_ref.abs().max().clamp_min(1e-12)
        assert (d - d_ref).abs().max() / scale < 1e-3, n


@pytest.mark.parametrize("name,D", [("DistMult", 64), ("ComplEx", 128), ("QMult", 64), ("OMult", 256), ("Keci", 96),
                                    ("TransE", 100)])
def test_negsample_step_matches_autograd(name, D):
    lr = 5.0
    ref, fused = _pair(name, D)
    tr = zipf_kg(600, 12, 5000, seed=2)
    ds = TriplePredictionDataset(tr, 600, 12, neg_sample_ratio=3, label_smoothing_rate=0.05).to(DEV)
    x, y = ds.make_batch(torch.arange(400, device=DEV))
    opt = torch.optim.SGD(ref.parameters(), lr=lr)
    loss_ref = ref.training_step((x, y))
    loss_ref.backward()
    opt.step()
    eng = FusedSampledEngine(fused, "NegSample", lr=lr, device=DEV, neg_ratio=3, label_smoothing=0.05, use_graph=False)
    loss = eng.step((x, y))
    eng.sync_to_model()
    assert abs(float(loss) - float(loss_ref)) < 1e-4 * abs(float(loss_ref))
    _compare_updates(ref, fused, lr)


def test_one_vs_sample_step_matches_autograd():
    lr = 5.0
    ref, fused = _pair("ComplEx", 64, scoring="1vsSample")
    tr = zipf_kg(600, 12, 5000, seed=3)
    ds = OnevsSample(tr, 600, 12, neg_sample_ratio=20, label_smoothing_rate=0.1).to(DEV)
    batch = ds.make_batch(torch.arange(256, device=DEV))
    opt = torch.optim.SGD(ref.parameters(), lr=lr)
    loss_ref = ref.training_step(batch)
    loss_ref.backward()
    opt.step()
    eng = FusedSampledEngine(fused, "1vsSample", lr=lr, device=DEV, use_graph=False)
    loss = eng.step(batch)
    eng.sync_to_model()
    assert abs(float(loss) - float(loss_ref)) < 1e-4 * abs(float(loss_ref))
    _compare_updates(ref, fused, lr)


def test_negsample_training_with_device_sampling_learns(umls_like_dir, tmp_path):
    """End to end through the trainer: graph replay, corruptions drawn inside the step, the model learns."""
    from dice_embeddings_b200 import Execute, Namespace
    rep = Execute(Namespace(dataset_dir=umls_like_dir, path_to_store_single_run=str(tmp_path / "run"),
                            model="ComplEx", scoring_technique="NegSample", neg_ratio=8, embedding_dim=32,
                            num_epochs=150, batch_size=1024, lr=0.1, gpus=0, kernel_backend="cuda",
                            trainer="torchCPUTrainer", eval_model="train_val_test")).start()
    assert rep["Train"]["MRR"] > 0.35, rep["Train"]


@pytest.mark.parametrize("kind,name", [(0, "Adam"), (2, "SGD")])
def test_sparse_rows_optimizer_updates_only_flagged_rows(kind, name):
    torch.manual_seed(0)
    rows, D = 1000, 128
    p = torch.randn(rows, D, device=DEV)
    g = torch.randn(rows, D, device=DEV)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    touched = (torch.rand(rows, device=DEV) < 0.3).to(torch.uint8)
    step = torch.zeros(1, dtype=torch.int64, device=DEV)
    ref = p.clone().requires_grad_(True)
    opt = torch.optim.Adam([ref], lr=0.01) if kind == 0 else torch.optim.SGD([ref], lr=0.01)
    ref.grad = g * touched[:, None].float()
    opt.step()
    p0, sel = p.clone(), touched.bool().clone()
    K.sparse_rows_optimizer(kind, p, g, m, v, None, touched, step, 0.01, 0.9, 0.999, 1e-8, 0.0)
    torch.cuda.synchronize()
    assert torch.equal(p[~sel], p0[~sel])                       # untouched rows are not even read
    assert torch.allclose(p[sel], ref.detach()[sel], atol=1e-5, rtol=1e-4)
    assert int(touched.sum()) == 0 and float(g[sel].abs().sum()) == 0.0 and float(g[~sel].abs().sum()) > 0


def test_uniform_int_into_column_block():
    cand = torch.full((300, 9), -1, dtype=torch.int64, device=DEV)
    K.uniform_int(cand[:, 1:], 50, seed=3)
    assert (cand[:, 0] == -1).all() and cand[:, 1:].min() >= 0 and cand[:, 1:].max() < 50
    flat = torch.empty(300 * 8, dtype=torch.int64, device=DEV)
    K.uniform_int(flat, 50, seed=3)
    assert torch.equal(flat.view(300, 8), cand[:, 1:])


# The drawn corruptions of the two-launch step: widths at the edges of the lane layouts (one, two and four floats per lane,
# several chunks), table sizes with and without chains (4 draws per row is the limit), groups split over several warps.
@pytest.mark.parametrize("name,D,NE,B,k", [
    ("DistMult", 4, 50, 33, 1), ("DistMult", 36, 4000, 700, 5), ("DistMult", 132, 4000, 700, 5), ("DistMult", 512, 900, 64, 3),
    ("ComplEx", 64, 4000, 333, 40), ("ComplEx", 72, 3000, 50, 100), ("ComplEx", 256, 100, 200, 9), ("ComplEx", 264, 3000, 65, 7),
    ("QMult", 64, 2000, 256, 3), ("QMult", 144, 2000, 100, 17), ("OMult", 256, 2000, 100, 9), ("OMult", 288, 2000, 31, 9),
    ("Keci", 96, 2000, 500, 10), ("Keci", 512, 2000, 100, 10), ("TransE", 100, 2000, 300, 6), ("TransE", 384, 60, 300, 6)])
def test_drawn_corruptions_match_autograd(name, D, NE, B, k):
    """fp32 sums of at most a few hundred terms in another order: 1e-4 of the largest gradient leaves a factor of 10."""
    gen = torch.Generator(device=DEV).manual_seed(D + NE)
    coins = set()
    for step in range(8):
        ref, fused = _pair(name, D, NE=NE)
        pos = torch.stack((torch.randint(0, NE, (B,), device=DEV, generator=gen),
                           torch.randint(0, 12, (B,), device=DEV, generator=gen),
                           torch.randint(0, NE, (B,), device=DEV, generator=gen)), 1)
        x = torch.zeros(B * (1 + k), 3, dtype=torch.int64, device=DEV)
        y = torch.zeros(B * (1 + k), device=DEV)
        K.neg_sample(pos, k, NE, 5, step, y, x=x, label_pos=0.9, label_neg=0.1)
        coin = bool((x[B:, 0] != pos[:, 0].repeat(k)).any())
        if coin in coins:
            continue
        coins.add(coin)
        ref = ref.double()
        loss_ref = torch.nn.functional.binary_cross_entropy_with_logits(ref(x), y.double())
        loss_ref.backward()
        eng = FusedSampledEngine(fused, "NegSample", lr=1.0, device=DEV, neg_ratio=k, label_smoothing=0.1, seed=5,
                                 use_graph=step % 2 == 0)
        eng.step_count.fill_(step)
        start = {n: p.detach().double().clone() for n, p in fused.named_parameters()}
        loss = eng.step((pos,))
        eng.sync_to_model()
        assert abs(float(loss) - float(loss_ref)) < 1e-5 * abs(float(loss_ref))
        for (n, p_ref), (_, p) in zip(ref.named_parameters(), fused.named_parameters()):
            if p_ref.grad is None:
                continue
            g = start[n] - p.detach().double()
            # the update w - lr g rounds w to 2^-24 of its size on top
            tol = 1e-4 * p_ref.grad.abs().max() + 2.0 ** -23 * start[n].abs().max()
            assert (g - p_ref.grad).abs().max() < tol, (n, coin)
        assert int(eng.touched.sum()) == 0 and int((eng.list_head != -1).sum()) == 0 and float(eng.gE.abs().sum()) == 0.0
        assert int(eng.step_count) == step + 1
    assert len(coins) == 2


@pytest.mark.parametrize("name,D,NE,B,k", [("TransE", 128, 5000, 300, 9), ("ComplEx", 64, 777, 40, 33), ("QMult", 256, 90, 64, 50)])
def test_sparse_update_of_drawn_tails(name, D, NE, B, k):
    """Row-wise sparse Adam over drawn tails: same rows, same values as the flagged-row optimiser on autograd's gradient."""
    ref, fused = _pair(name, D, NE=NE)
    gen = torch.Generator(device=DEV).manual_seed(3)
    pos = torch.stack((torch.randint(0, NE, (B,), device=DEV, generator=gen), torch.randint(0, 12, (B,), device=DEV, generator=gen),
                       torch.randint(0, NE, (B,), device=DEV, generator=gen)), 1)
    cand = torch.zeros(B, 1 + k, dtype=torch.int64, device=DEV)
    cand[:, 0] = pos[:, 2]
    step = torch.full((1,), 7, dtype=torch.int64, device=DEV)
    K.uniform_int(cand[:, 1:], NE, 11, 0, step=step)
    x = torch.stack((pos[:, :1].expand(-1, 1 + k), pos[:, 1:2].expand(-1, 1 + k), cand), 2).reshape(-1, 3)
    y = torch.full((B, 1 + k), 0.1, device=DEV)
    y[:, 0] = 0.9
    loss_ref = torch.nn.functional.binary_cross_entropy_with_logits(ref(x), y.reshape(-1))
    loss_ref.backward()
    E, R = fused.entity_embeddings.weight.data, fused.relation_embeddings.weight.data
    z = torch.zeros_like
    mE = 1e-3 * torch.randn(E.shape, device=DEV, generator=gen)
    vE = 1e-6 * (1 + torch.rand(E.shape, device=DEV, generator=gen))
    touched, head = torch.zeros(NE, dtype=torch.uint8, device=DEV), torch.full((NE,), -1, dtype=torch.int32, device=DEV)
    loss_acc, loss_out = torch.zeros(1, dtype=torch.float64, device=DEV), torch.zeros(1, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want_p, want_m, want_v = E.clone(), mE.clone(), vE.clone()
    flags = torch.zeros(NE, dtype=torch.uint8, device=DEV)
    flags[cand.reshape(-1)] = 1
    flags[pos[:, 0]] = 1
    K.sparse_rows_optimizer(0, want_p, ref.entity_embeddings.weight.grad.clone(), want_m, want_v, None, flags, step, 0.01, 0.9,
                            0.999, 1e-8, 0.0)
    s = K.SampledStep(K.MODEL_CODE[name], name == "QMult", "tails", B, 1 + k, E, z(E), mE, vE, touched, head, R, z(R), z(R), z(R),
                      None, None, None, None, 0, True, 11, 0.9, 0.1, 1.0 / (B * (1 + k)), float(getattr(fused, "margin", 0.0)),
                      float(getattr(fused, "_eps", 0.0)), step, loss_acc, loss_out, status, NE)
    s.launch(0.01, 0.9, 0.999, 1e-8, 0.0, pos=pos)
    torch.cuda.synchronize()
    assert int(status) == 0 and int(step) == 8 and abs(float(loss_out) - float(loss_ref)) < 1e-5 * float(loss_ref)
    # gradients agree to 1e-4 of the largest (sums in another order); moments and weights follow from them
    g = float(ref.entity_embeddings.weight.grad.abs().max())
    assert (mE - want_m).abs().max() < 1e-5 * g + 1e-9
    assert (vE - want_v).abs().max() < 1e-6 * g * g + 1e-12
    assert (E - want_p).abs().max() < 0.01 * (1e-5 * g + 1e-9) / 1e-3 * 10 + 1e-6
    assert int(touched.sum()) == 0 and int((head != -1).sum()) == 0


@pytest.mark.parametrize("name,D,C", [("DistMult", 64, 6), ("DistMult", 512, 2), ("ComplEx", 128, 33), ("TransE", 100, 5), ("QMult", 256, 1),
                                      ("OMult", 512, 3)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_row_that_is_not_a_number_stays_where_it_is(name, D, C, bad):
    """Entities that no triple of the batch names do not reach it, whatever they hold: candidate counts that leave part of the
    rows in flight empty."""
    _, m = _pair(name, D, NE=100, scoring="1vsSample")
    with torch.no_grad():
        m.entity_embeddings.weight[0] = bad
        m.entity_embeddings.weight[99] = bad
    eng = FusedSampledEngine(m, "1vsSample", lr=1.0, device=DEV, use_graph=False)
    x = torch.stack((torch.randint(1, 99, (30,), device=DEV), torch.randint(0, 12, (30,), device=DEV)), 1)
    loss = eng.step((x, torch.randint(1, 99, (30, C), device=DEV), torch.rand(30, C, device=DEV).round()))
    assert torch.isfinite(loss) and torch.isfinite(eng.E[1:99]).all() and torch.isfinite(eng.R).all()


@pytest.mark.parametrize("engine", ["1vsSample", "NegSample", "one rank"])
def test_further_columns_of_a_batch_are_not_looked_at(engine):
    """Index rows with more columns than the step needs: the same step as on the columns it needs."""
    import torch.distributed as dist
    st = "NegSample" if engine == "NegSample" else "1vsSample"
    pair = _pair("ComplEx", 64, scoring=st)
    gen = torch.Generator(device=DEV).manual_seed(0)
    x = torch.randint(0, 12, (30, 5), device=DEV, generator=gen)
    y = torch.rand(30, 1 if st == "NegSample" else 7, device=DEV, generator=gen).round()
    rest = (y[:, 0],) if st == "NegSample" else (torch.randint(0, 600, (30, 7), device=DEV, generator=gen), y)
    out = []
    try:
        if engine == "one rank":
            from dice_embeddings_b200.parallel.sharded_sampled import ShardedSampledEngine
            dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=DEV)
        for m, cols in zip(pair, (5, 3 if st == "NegSample" else 2)):
            if engine == "one rank":
                eng = ShardedSampledEngine(m, st, batch_size=30, lr=5.0, device=DEV, use_graph=False)
            else:
                eng = FusedSampledEngine(m, st, lr=5.0, device=DEV, use_graph=False)
            out.append((float(eng.step((x[:, :cols].contiguous(), *rest))), eng.E.clone()))
        assert abs(out[0][0] - out[1][0]) < 1e-6 and torch.allclose(out[0][1], out[1][1], atol=1e-5)
    finally:
        if dist.is_initialized():
            dist.destroy_process_group()
