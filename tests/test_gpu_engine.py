"""The fused training step against a PyTorch fp32 implementation of the same step."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

from dice_embeddings_b200.data.datasets import KvsAll, OnevsAllDataset
from dice_embeddings_b200.data.synthetic import zipf_kg
from dice_embeddings_b200.models import initialize_model
from dice_embeddings_b200.ops.fused_step import FusedKvsAllEngine, build_fused_engine
from dice_embeddings_b200.ops.hybrid_step import ExternalQueryEngine

DEV = torch.device("cuda:0")


def _make(name, D, optim, lr, NE=700, NR=15, smoothing=0.1, seed=0, scoring="KvsAll"):
    tr = zipf_kg(NE, NR, 4000, seed=seed)
    ds = (KvsAll(tr, NE, NR, label_smoothing_rate=smoothing) if scoring == "KvsAll" else OnevsAllDataset(tr, NE)).to(DEV)
    torch.manual_seed(seed)
    args = dict(model=name, embedding_dim=D, num_entities=NE, num_relations=NR, optim=optim, learning_rate=lr,
                scoring_technique=scoring, p=0, q=1)
    m1, _ = initialize_model(dict(args))
    m2, _ = initialize_model(dict(args))
    m2.load_state_dict(m1.state_dict())
    for m in (m1, m2):
        m.to(DEV)
        with torch.no_grad():
            m.entity_embeddings.weight.mul_(0.3)
            m.relation_embeddings.weight.mul_(0.3)
            if name == "Keci":
                m.q_coefficients.weight.fill_(0.5)
    return ds, m1, m2


@pytest.mark.parametrize("name,label_mode", [("DistMult", "mask"), ("ComplEx", "mask"), ("ComplEx", "sparse"),
                                             ("QMult", "mask"), ("OMult", "sparse"), ("Keci", "mask")])
@pytest.mark.parametrize("D", [64, 256])
def test_one_sgd_step_matches_autograd(name, label_mode, D):
    """With SGD the parameter change is the gradient itself, so this checks every gradient path."""
    lr = 50.0  # gradients of a mean over B x |E| logits are tiny
    ds, ref, fused = _make(name, D, "SGD", lr)
    B = 384
    idx = torch.randperm(len(ds), device=DEV)[:B]
    x, y = ds.make_batch(idx)
    opt = ref.configure_optimizers()
    loss_ref = ref.training_step((x, y))
    loss_ref.backward()
    opt.step()
    eng = FusedKvsAllEngine(fused, ds, batch_size=B, lr=lr, device=DEV, use_graph=False, label_mode=label_mode)
    loss = eng.step((x, idx))
    eng.sync_to_model()
    assert abs(float(loss) - float(loss_ref.detach())) < 1e-2 * abs(float(loss_ref.detach()))
    for (n, p_ref), (_, p) in zip(ref.named_parameters(), fused.named_parameters()):
        upd_ref = p_ref.detach() - 0  # after step
        # compare parameter *changes*: start values are identical copies
        start = p_ref.detach() + lr * p_ref.grad
        d_ref, d = upd_ref - start, p.detach() - start
        scale = d_ref.abs().max().clamp_min(1e-12)
        assert (d - d_ref).abs().max() / scale < 5e-2, n


@pytest.mark.parametrize("name,extra", [("ConEx", {}), ("AConEx", {}), ("ConvQ", {}), ("AConvO", {}), ("DualE", {}),
                                        ("ComplEx", {"normalization": "LayerNorm"}),
                                        ("QMult", {"normalization": "BatchNorm1d"}),
                                        ("Keci", {"p": 1, "q": 2}), ("DeCaL", {"p": 3, "q": 3, "r": 1}),
                                        ("TransE", {}), ("CoKE", {})])
@pytest.mark.parametrize("D", [64, 256])
def test_external_query_engine_matches_autograd(name, extra, D):
    """Models whose query vector comes out of PyTorch modules (convolutional gates, normalisers, dual quaternions),
    models with a per-query scalar next to the dot product (general Clifford algebras) and the distance model: one SGD step through the tensor-core scoring function against the same step in plain autograd on dense labels."""
    from dice_embeddings_b200.ops.hybrid_step import ExternalQueryEngine, build_hybrid_engine, hybrid_supported
    lr = 50.0
    NE, NR = 700, 15
    tr = zipf_kg(NE, NR, 4000, seed=0)
    ds = KvsAll(tr, NE, NR, label_smoothing_rate=0.1).to(DEV)
    torch.manual_seed(0)
    args = dict(model=name, embedding_dim=D, num_entities=NE, num_relations=NR, optim="SGD", learning_rate=lr,
                scoring_technique="KvsAll", num_of_output_channels=2, kernel_size=3, **extra)
    ref, _ = initialize_model(dict(args))
    hyb, _ = initialize_model(dict(args))
    hyb.load_state_dict(ref.state_dict())
    for m in (ref, hyb):
        m.to(DEV)
        with torch.no_grad():
            m.entity_embeddings.weight.mul_(0.3)
            m.relation_embeddings.weight.mul_(0.3)
            for n, p in m.named_parameters():
                if "coefficients" in n:
                    p.fill_(0.7)           # the interaction terms (and with them the per-query bias) are switched on
        m.train()
        for mod in m.modules():            # the transformer's dropout would draw different masks in the two runs
            if isinstance(mod, torch.nn.Dropout):
                mod.p = 0.0
            if isinstance(getattr(mod, "dropout", None), float):
                mod.dropout = 0.0
    assert hybrid_supported(hyb)
    B = 384
    idx = torch.randperm(len(ds), device=DEV)[:B]
    x, y = ds.make_batch(idx)
    start = {n: p.detach().clone() for n, p in ref.named_parameters()}
    opt = ref.configure_optimizers()
    loss_ref = ref.training_step((x, y))
    loss_ref.backward()
    opt.step()
    eng = build_hybrid_engine(hyb, ds, type("A", (), dict(scoring_technique="KvsAll", batch_size=B, lr=lr))(), DEV)
    assert isinstance(eng, ExternalQueryEngine)
    loss = eng.step((x, idx))
    eng.sync_to_model()
    assert abs(float(loss) - float(loss_ref.detach())) < 1e-2 * abs(float(loss_ref.detach()))
    moved = 0
    for (n, p_ref), (_, p) in zip(ref.named_parameters(), hyb.named_parameters()):
        d_ref, d = p_ref.detach() - start[n], p.detach() - start[n]
        scale = d_ref.abs().max()
        if n == "conv2d.bias" or scale < 1e-5 * start[n].abs().max().clamp_min(1e-3):
            continue   # the batch norm behind the convolution removes its bias: that gradient is rounding noise
        moved += 1
        assert (d - d_ref).abs().max() < 6e-2 * scale + 1e-6, n
    assert moved >= 2


@pytest.mark.parametrize("optim", ["Adam", "Adopt"])
def test_loss_trajectory_with_graph_replay(optim):
    ds, ref, fused = _make("ComplEx", 128, optim, 0.02)
    B = 256
    opt = ref.configure_optimizers()
    eng = FusedKvsAllEngine(fused, ds, batch_size=B, lr=0.02, device=DEV, use_graph=True)
    g = torch.Generator(device="cpu").manual_seed(0)
    ref_losses, losses = [], []
    for _ in range(6):
        idx = torch.randperm(len(ds), generator=g)[:B].to(DEV)
        x, y = ds.dense_batch(idx)
        opt.zero_grad()
        l = ref.training_step((x, y))
        l.backward()
        opt.step()
        ref_losses.append(float(l.detach()))
        losses.append(float(eng.step((x, idx))))
    eng.sync_to_model()
    for a, b in zip(losses, ref_losses):
        assert abs(a - b) < 3e-2 * abs(b), (losses, ref_losses)
    assert losses[-1] < losses[0]


def test_one_vs_all_and_host_step():
    ds, ref, fused = _make("DistMult", 64, "Adam", 0.05, scoring="1vsAll")
    B = 200
    idx = torch.arange(B, device=DEV)
    x, y = ds.make_batch(idx)
    loss_ref = float(ref.training_step((x, y)).detach())
    eng = FusedKvsAllEngine(fused, ds, batch_size=B, lr=0.05, device=DEV)
    loss = eng.step_from_host(x.cpu().pin_memory(), idx.cpu().pin_memory())
    assert abs(loss - loss_ref) < 1e-2 * abs(loss_ref)


def test_trainer_uses_fused_engine(tmp_path):
    from dice_embeddings_b200 import Execute, KGE, Namespace
    from dice_embeddings_b200.data.synthetic import make_planted_kg
    kg = make_planted_kg(str(tmp_path / "kg"), num_entities=300, num_relations=10, seed=1)
    a = Namespace(dataset_dir=kg, model="ComplEx", scoring_technique="KvsAll", embedding_dim=64, num_epochs=100,
                  batch_size=256, lr=0.1, optim="Adam", path_to_store_single_run=str(tmp_path / "run"), gpus=0,
                  kernel_backend="cuda", trainer="torchCPUTrainer")
    rep = Execute(a).start()
    assert rep["Train"]["MRR"] > 0.9
    k = KGE(path=str(tmp_path / "run"))
    assert len(k.predict_topk(h=[next(iter(k.entity_to_idx))], r=[next(iter(k.relation_to_idx))], topk=3)[0]) == 3


@pytest.mark.parametrize("model,extra", [("TransE", {}), ("Keci", {"p": 1, "q": 2}), ("ConEx", {"num_of_output_channels": 2})])
def test_trainer_uses_external_query_engine(tmp_path, model, extra):
    """The distance model, a Clifford model with per-query scalar terms and a convolutional model train through
    ``Execute`` on the tensor-core scoring function and learn the planted graph."""
    from dice_embeddings_b200 import Execute, Namespace
    from dice_embeddings_b200.data.synthetic import make_planted_kg
    from dice_embeddings_b200.ops.hybrid_step import ExternalQueryEngine
    kg = make_planted_kg(str(tmp_path / "kg"), num_entities=300, num_relations=10, seed=1)
    a = Namespace(dataset_dir=kg, model=model, scoring_technique="KvsAll", embedding_dim=64, num_epochs=150,
                  batch_size=256, lr=0.05, optim="Adam", path_to_store_single_run=str(tmp_path / "run"), gpus=0,
                  kernel_backend="cuda", trainer="torchCPUTrainer", **extra)
    ex = Execute(a)
    rep = ex.start()
    assert isinstance(ex.trainer.trainer.engine, ExternalQueryEngine)
    assert rep["Train"]["MRR"] > 0.5, rep["Train"]


def test_pipelined_host_steps_return_the_same_losses():
    ds, m1, m2 = _make("ComplEx", 64, "Adam", 0.05)
    B = 256
    e1 = FusedKvsAllEngine(m1, ds, batch_size=B, lr=0.05, device=DEV)
    e2 = FusedKvsAllEngine(m2, ds, batch_size=B, lr=0.05, device=DEV)
    g = torch.Generator().manual_seed(3)
    pairs = ds.train_data.cpu()
    a, b = [], []
    for _ in range(6):
        idx = torch.randperm(len(ds), generator=g)[:B]
        x, dp = pairs[idx].contiguous().pin_memory(), idx.contiguous().pin_memory()
        a.append(e1.step_from_host(x, dp))
        b.append(e2.step_from_host_pipelined(x, dp))
    b = b[1:] + [e2.last_loss()]
    assert all(abs(u - v) < 1e-6 * max(1.0, abs(u)) for u, v in zip(a, b)), (a, b)


@pytest.mark.parametrize("name,optim", [("ConEx", "Adam"), ("TransE", "AdamW"), ("DualE", "SGD"), ("ConvQ", "Adopt")])
def test_external_query_step_from_a_graph_equals_plain_launches(name, optim):
    """Same losses and weights from replayed and plain steps: two batch sizes, a learning-rate change, evaluation mode in
    between (sums with atomics in another order: 1e-4 of the weights' change)."""
    engines = []
    for use_graph in (True, False):
        torch.manual_seed(0)
        tr = zipf_kg(700, 9, 6000, seed=1)
        ds = KvsAll(tr, 700, 9, label_smoothing_rate=0.1).to(DEV)
        model, _ = initialize_model(dict(model=name, embedding_dim=64, num_entities=700, num_relations=9, optim=optim,
                                         learning_rate=0.01, scoring_technique="KvsAll", num_of_output_channels=4, kernel_size=3))
        model = model.to(DEV).train()
        with torch.no_grad():
            model.entity_embeddings.weight.mul_(0.3)
            model.relation_embeddings.weight.mul_(0.3)
        engines.append((ExternalQueryEngine(model, ds, batch_size=256, lr=1e-3, device=DEV, use_graph=use_graph), ds, model))
    start = [p.detach().clone() for p in engines[0][2].parameters()]
    losses = [[], []]
    for step in range(12):
        n = 256 if step % 3 else 199
        for k, (eng, ds, model) in enumerate(engines):
            if step == 8:
                eng.optimizer_view().param_groups[0]["lr"] = 5e-4
            idx = torch.arange(step * 7, step * 7 + n, device=DEV) % len(ds)
            batch = ds.make_batch(idx)
            losses[k].append(eng.step((batch[0], idx)))
    for eng, _, _ in engines:
        eng.sync_to_model()
    assert len(engines[0][0]._graphs) > 0 or optim == "Adopt"
    a, b = (torch.stack(x) for x in losses)
    assert len({x.data_ptr() for x in losses[0]}) == 12 and a.unique().numel() > 6   # every step's loss is its own tensor
    assert torch.allclose(a, b, rtol=1e-4), (a, b)
    # Adam divides a gradient by its own size: an element whose gradient is rounding noise (atomics in another order) may move
    # by the learning rate either way, 2 * (8 * 1e-3 + 4 * 5e-4) = 0.02 at most over the run.  Few elements are like that,
    # so the 2-norm of the change is compared; the bias ahead of the batch normalisation is (its true gradient is zero),
    # and with it the running mean.
    for s, (name, p), q in zip(start, engines[0][2].named_parameters(), engines[1][2].parameters()):
        if name.endswith("conv2d.bias"):
            assert (p - q).abs().max() <= 0.02
            continue
        assert (p - q).norm() <= 1e-2 * (q - s).norm() + 1e-6, (name, float((p - q).norm()), float((q - s).norm()))
    for (n1, x), (_, y) in zip(engines[0][2].named_buffers(), engines[1][2].named_buffers()):
        assert torch.allclose(x.float(), y.float(), rtol=1e-3, atol=0.02 if n1.endswith("running_mean") else 1e-5), n1


def test_external_query_step_with_hooks_runs_as_plain_launches():
    tr = zipf_kg(300, 5, 2000, seed=1)
    ds = KvsAll(tr, 300, 5).to(DEV)
    model, _ = initialize_model(dict(model="ConEx", embedding_dim=64, num_entities=300, num_relations=5, optim="Adam",
                                     learning_rate=0.01, scoring_technique="KvsAll", num_of_output_channels=4, kernel_size=3))
    model = model.to(DEV).train()
    eng = ExternalQueryEngine(model, ds, batch_size=64, lr=0.01, device=DEV)
    idx = torch.arange(64, device=DEV)
    for _ in range(3):
        eng.step(ds.make_batch(idx)[:1] + (idx,))
    assert len(eng._graphs) == 1
    triples = torch.cat((ds.make_batch(idx)[0][:, :2], idx[:, None] % 300), 1)      # further columns are not looked at
    assert torch.isfinite(eng.step((triples, idx))) and len(eng._graphs) == 1
    calls = []
    handle = model.fc1.register_forward_hook(lambda *a: calls.append(1))
    eng.step(ds.make_batch(idx)[:1] + (idx,))
    packed = []
    handle.remove()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(1) or t, lambda t: t):
        eng.step(ds.make_batch(idx)[:1] + (idx,))
    assert len(calls) == 1 and packed


@pytest.mark.parametrize("what", ["momentum", "eps", "dropout", "margin", "function", "betas"])
def test_host_values_changed_after_a_capture_take_effect(what):
    """Replay fixes what a step reads on the host: a change of such a value gives the same state as plain launches do (atomics in
    another order: 1e-3), here far from the state without the change."""
    out = []
    for use_graph, change in ((True, True), (False, True), (False, False)):
        torch.manual_seed(0)
        name = "TransE" if what == "margin" else "ConEx"
        ds = KvsAll(zipf_kg(300, 9, 3000, seed=1), 300, 9, label_smoothing_rate=0.1).to(DEV)
        model, _ = initialize_model(dict(model=name, embedding_dim=64, num_entities=300, num_relations=9, optim="SGD",
                                         learning_rate=0.01, scoring_technique="KvsAll", num_of_output_channels=4, kernel_size=3))
        model = model.to(DEV).train()
        eng = ExternalQueryEngine(model, ds, batch_size=128, lr=0.05, device=DEV, use_graph=use_graph)
        idx = torch.arange(128, device=DEV)
        batch = (ds.make_batch(idx)[0], idx)
        for _ in range(3):
            eng.step(batch)
        if change:
            if what == "momentum":
                model.bn_conv2d.momentum = 0.9
            elif what == "eps":
                model.bn_conv2d.eps = 0.5
            elif what == "dropout":
                model.input_dp_ent_real.p = 1.0
            elif what == "margin":
                eng.margin += 2.0
            elif what == "function":
                model.fc1.forward = lambda x, fc=model.fc1: torch.nn.functional.linear(x, fc.weight, fc.bias) + 1.0
            else:
                eng.weight_decay, eng.betas = 0.3, (0.5, 0.9)
        for _ in range(3):
            loss = eng.step(batch)
        out.append(torch.cat([loss.reshape(1), eng.E.flatten()] + [b.float().flatten() for b in model.buffers()]))
        assert len(eng._graphs) == ((2 if change else 1) if use_graph else 0)
    size = (out[1] - out[2]).norm()
    assert (out[0] - out[1]).norm() < 1e-3 * out[1].norm() and (out[0] - out[1]).norm() < 0.1 * size, (what, size)


def _small_engine(**kw):
    ds = KvsAll(zipf_kg(300, 9, 3000, seed=1), 300, 9, label_smoothing_rate=0.1).to(DEV)
    model, _ = initialize_model(dict(model="ConEx", embedding_dim=64, num_entities=300, num_relations=9, optim="Adam",
                                     learning_rate=0.01, scoring_technique="KvsAll", num_of_output_channels=4, kernel_size=3))
    eng = ExternalQueryEngine(model.to(DEV).train(), ds, batch_size=128, lr=0.05, device=DEV, **kw)
    idx = torch.arange(128, device=DEV)
    eng.plain, step = 0, eng._step

    def counted(*a):
        eng.plain += 1
        return step(*a)
    eng._step = counted
    return eng, (ds.make_batch(idx)[0], idx)


def test_replay_follows_a_learning_rate_schedule():
    """More rates than graphs are kept: every rate is replayed in the end, the oldest graphs go, and a rate that stays for a
    few steps only does not push out one in use."""
    eng, batch = _small_engine()
    view = eng.optimizer_view().param_groups[0]
    late = eng.STEPS_BEFORE_REPLACING
    for epoch in range(eng.MAX_GRAPHS + 3):
        view["lr"] = 0.05 / (epoch + 1)
        eng.plain = 0
        for _ in range(late + 10):
            assert torch.isfinite(eng.step(batch))
        assert eng.plain == (2 if epoch < eng.MAX_GRAPHS else late + 1), epoch      # the capture runs the step's host side once
        assert len(eng._graphs) == min(epoch + 1, eng.MAX_GRAPHS)
    kept = list(eng._graphs)
    for i in range(2 * eng.MAX_KINDS):                  # a rate of its own for every step
        view["lr"] = 1e-3 / (i + 1)
        eng.step(batch)
    assert list(eng._graphs) == kept and len(eng._seen) == eng.MAX_KINDS
    view["lr"] = 0.05 / (eng.MAX_GRAPHS + 3)
    eng.plain = 0
    eng.step(batch)
    assert eng.plain == 0


def test_a_failed_capture_is_reported_and_the_step_goes_on(caplog):
    """The process is as it was before: the caller's stream is current, random numbers (here of a dropout) can be drawn and follow
    the seed, memory can be had and given back, and another engine captures and replays its steps."""
    eng, batch = _small_engine()
    eng.step(batch)
    forward = eng.model.fc1.forward
    eng.model.input_dp_ent_real.p = 0.3

    def waits(x):
        float(x.detach().sum())                         # a copy to the host: not allowed in a capture
        return forward(x)
    eng.model.fc1.forward = waits
    stream = torch.cuda.current_stream()
    for _ in range(4):
        assert torch.isfinite(eng.step(batch))
        assert torch.cuda.current_stream() == stream
    assert not eng._graphs and not eng.use_graph and sum("capture failed" in r.message for r in caplog.records) == 1
    draws = []
    for _ in range(2):
        torch.manual_seed(5)
        draws.append(torch.rand(1000, device=DEV))
    assert torch.equal(*draws) and 0.4 < float(draws[0].mean()) < 0.6
    del draws
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    other, batch = _small_engine()
    other.model.input_dp_ent_real.p = 0.3
    other.optimizer_view().param_groups[0]["lr"] = 0.0      # the same weights throughout: only the dropout differs
    losses = [float(other.step(batch)) for _ in range(5)]
    assert len(other._graphs) == 1 and len(set(losses)) == 5 and all(x == x for x in losses)
