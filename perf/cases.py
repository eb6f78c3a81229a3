"""The work that users of this framework have it do on one GPU, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` names the ones that stand for everyday use, ``draw(rng)`` gives further
ones of the same ranges, ``prepare`` makes what a user's program holds before the call (weights, data set, engine or
ranker, a batch on the device) from a seed, ``run`` is one pass through the public entry point, ``work`` the bytes and
operations that pass cannot do without and ``tolerance`` how far another correct implementation may be off.

Six kinds of work:

* ``kvsall``     a training step against all entities (KvsAll / 1vsAll) of a model whose query is an algebra product:
                 ``FusedKvsAllEngine.step``, the call of the single-device trainer per batch;
* ``hybrid``     the same for models whose query comes out of PyTorch modules or whose score is a distance:
                 ``ExternalQueryEngine.step``;
* ``sampled``    a training step on sampled candidates with a dense optimiser (NegSample, 1vsSample, KvsSample):
                 ``FusedSampledEngine.step``;
* ``rowsparse``  the same on a table of millions of rows with the row-wise sparse optimiser (one rank of the sharded
                 trainer): ``ShardedSampledEngine.step``;
* ``evaluate``   filtered tail ranks of a model as the evaluator asks for them: ``tail_ranks`` from index triples on the
                 host to ranks on the host;
* ``rank`` / ``topk``  ranks and best tails of a batch of query vectors against a resident table: ``FusedRanker``.

The training states are those of a run that has been going for a while: the engine has taken its first steps (its launch
graph exists), the moments have the size of the gradients, the step counter is past the start.  Gradients can be read off
the returned first moments.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda:0"


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest training step in use: UMLS-shaped graph, the wide embedding and small batch of its usual runs
        dict(name="kvsall small", kind="kvsall", model="Keci", technique="KvsAll", entities=135, relations=46,
             triples=5216, dim=256, batch=32, optim="Adam"),
        # the headline benchmark: FB15k-237-shaped graph, label smoothing, Adam
        dict(name="kvsall headline", kind="kvsall", model="ComplEx", technique="KvsAll", entities=14541,
             relations=237, triples=272115, dim=256, batch=4096, optim="Adam"),
        # an odd vocabulary and a ragged batch (the last one of an epoch) with one positive per query
        dict(name="1vsall ragged", kind="kvsall", model="QMult", technique="1vsAll", entities=40559, relations=22,
             triples=86835, dim=128, batch=1111, optim="AdamW"),
        # a table of millions of rows: labels as a sparse correction instead of masks
        dict(name="kvsall large", kind="kvsall", model="DistMult", technique="KvsAll", entities=2000000,
             relations=1000, triples=1000000, dim=256, batch=8192, optim="Adam"),
        # convolutional gate in autograd, scoring and table update in the kernels
        dict(name="conex", kind="hybrid", model="ConEx", entities=14541, relations=237, triples=272115, dim=256,
             batch=1024, channels=8),
        # YAGO3-10-shaped negative sampling: ten corruptions per positive, batch 10 000, dense Adam
        dict(name="negsample", kind="sampled", model="Keci", technique="NegSample", entities=123182, relations=37,
             dim=128, batch=10000, negatives=10, optim="Adam"),
        # given candidate lists per (head, relation) pair
        dict(name="kvssample", kind="sampled", model="ComplEx", technique="KvsSample", entities=14541, relations=237,
             dim=256, batch=1024, negatives=99, optim="Adam"),
        # 128 corrupted tails per positive on a table whose rows are touched sparsely
        dict(name="negsample row-sparse", kind="rowsparse", model="TransE", entities=5000000, relations=5000, dim=128,
             batch=32768, negatives=128),
        # filtered link prediction of a test split at the headline shape, host to host
        dict(name="evaluate", kind="evaluate", model="ComplEx", entities=14541, relations=237, triples=272115,
             dim=256, queries=20466, batch=4096),
        # filtered ranks against a table of millions of rows
        dict(name="rank large", kind="rank", entities=2000000, dim=256, queries=8192, filters=16),
        # batch prediction and a single interactive question
        dict(name="topk large", kind="topk", entities=2000000, dim=256, queries=1024, k=10),
        dict(name="topk one", kind="topk", entities=14541, dim=256, queries=1, k=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kvsall", "kvsall", "hybrid", "sampled", "rowsparse", "evaluate", "rank", "topk"])
    if kind == "kvsall":
        dim = rng.choice([64, 128, 256])
        batch = _log(rng, 32, 8192)
        entities = _log(rng, 135, 1000000)
        return dict(kind=kind, model=rng.choice(["DistMult", "ComplEx", "QMult", "OMult", "Keci"]),
                    technique=rng.choice(["KvsAll", "KvsAll", "1vsAll"]), entities=entities,
                    relations=_log(rng, 11, 1000), triples=min(max(3 * batch, 8 * entities), 300000 + entities),
                    dim=dim, batch=batch, optim=rng.choice(["Adam", "Adam", "AdamW", "Adopt"]))
    if kind == "hybrid":
        entities = _log(rng, 1000, 50000)
        return dict(kind=kind, model=rng.choice(["ConEx", "AConEx", "ConvQ", "TransE", "Keci12", "DualE"]),
                    entities=entities, relations=_log(rng, 11, 1000), triples=8 * entities + 20000,
                    dim=rng.choice([64, 128, 256]), batch=_log(rng, 128, 4096), channels=rng.choice([2, 4, 8]))
    if kind == "sampled":
        batch = _log(rng, 32, 16384)
        return dict(kind=kind, model=rng.choice(["TransE", "DistMult", "ComplEx", "Keci", "QMult"]),
                    technique=rng.choice(["NegSample", "NegSample", "1vsSample", "KvsSample"]),
                    entities=_log(rng, 135, 200000), relations=_log(rng, 11, 1000),
                    dim=rng.choice([32, 64, 128, 256]), batch=batch,
                    negatives=_log(rng, 1, min(128, 200000 // batch)), optim=rng.choice(["Adam", "Adam", "AdamW", "Adopt"]))
    if kind == "rowsparse":
        return dict(kind=kind, model=rng.choice(["TransE", "DistMult", "ComplEx", "QMult"]),
                    entities=_log(rng, 200000, 5000000), relations=_log(rng, 11, 5000), dim=rng.choice([64, 128]),
                    batch=_log(rng, 1024, 32768), negatives=_log(rng, 8, 128))
    if kind == "evaluate":
        entities = _log(rng, 135, 40000)
        return dict(kind=kind, model=rng.choice(["DistMult", "ComplEx", "QMult"]), entities=entities,
                    relations=_log(rng, 11, 500), triples=min(12 * entities, 300000), dim=rng.choice([32, 64, 128, 256]),
                    queries=min(_log(rng, 500, 20466), 6 * entities), batch=rng.choice([1024, 2048, 4096]))
    if kind == "rank":
        return dict(kind=kind, entities=_log(rng, 20000, 2000000), dim=rng.choice([64, 128, 256]),
                    queries=_log(rng, 64, 8192), filters=_log(rng, 1, 64))
    return dict(kind=kind, entities=_log(rng, 2000, 2000000), dim=rng.choice([64, 128, 256]),
                queries=_log(rng, 1, 1024), k=rng.choice([1, 3, 10, 32]))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (2 ** 62))


def _graph(case, seed):
    """Distinct index triples.  Graphs of ordinary size have Zipf degrees; a table of millions of rows gets its heavy
    tail from the third power of a uniform number (far cheaper to draw)."""
    from dice_embeddings_b200.data.synthetic import zipf_kg
    ne, nr, nt = case["entities"], case["relations"], case["triples"]
    if ne <= 50000:
        return zipf_kg(ne, nr, nt, 1.1, 1.3, seed=seed % (2 ** 31))
    rng = np.random.default_rng(seed)
    e = np.minimum((ne * rng.random((nt, 2)) ** 3).astype(np.int64), ne - 1)
    return np.stack([e[:, 0], rng.integers(0, nr, nt), e[:, 1]], axis=1)


def _model(name, case, optim, technique, **extra):
    from dice_embeddings_b200.models import initialize_model
    args = dict(model=name, embedding_dim=case["dim"], num_entities=case["entities"], num_relations=case["relations"],
                optim=optim, learning_rate=0.01, scoring_technique=technique, p=0, q=1, **extra)
    with torch.device(DEV):
        return initialize_model(args)[0]


def _load(param, gen, scale):
    param.normal_(generator=gen).mul_(scale)


def _load_moments(m, v, gen, g):
    """Moments of a run under way: gradients of size ``g`` with the usual spread."""
    m.normal_(generator=gen).mul_(0.3 * g)
    v.uniform_(0.5, 1.5, generator=gen).mul_(g * g)


@torch.no_grad()
def _resume(engine, case, gen, g_ent, g_rel):
    """Weights and optimiser state of a run under way, loaded into an engine that has taken its first steps."""
    _load(engine.E, gen, 0.25)
    if hasattr(engine, "R"):
        _load(engine.R, gen, 0.25)
        if engine.coeff is not None:
            engine.coeff.fill_(0.7)
            if getattr(engine, "mC", None) is not None:
                engine.mC.fill_(g_rel)
                engine.vC.fill_(g_rel * g_rel)
        _load_moments(engine.mR, engine.vR, gen, g_rel)
    _load_moments(engine.mE, engine.vE, gen, g_ent)
    engine.step_count.fill_(200)


def _prepare_kvsall(case, seed):
    from dice_embeddings_b200.data.datasets import KvsAll, OnevsAllDataset
    from dice_embeddings_b200.ops import kernels
    from dice_embeddings_b200.ops.fused_step import FusedKvsAllEngine
    gen = _gen(seed)
    triples = _graph(case, seed)
    if case["technique"] == "KvsAll":
        ds = KvsAll(triples, case["entities"], case["relations"], label_smoothing_rate=0.1).to(DEV)
    else:
        ds = OnevsAllDataset(triples, case["entities"]).to(DEV)
    model = _model(case["model"], case, case["optim"], case["technique"])
    engine = FusedKvsAllEngine(model, ds, batch_size=case["batch"], lr=0.01, weight_decay=0.0, device=DEV)
    n = len(ds)
    idx = torch.randperm(n, device=DEV, generator=gen)[:case["batch"]]
    batch = ds.make_batch(idx)
    engine.step(batch)
    g_ent = 0.1 / (math.sqrt(case["batch"]) * case["entities"])
    _resume(engine, case, gen, g_ent, 10 * g_ent)
    kernels.cast_bf16(engine.E, engine.E_bf16)
    return dict(engine=engine, batch=batch)


def _prepare_hybrid(case, seed):
    from dice_embeddings_b200.data.datasets import KvsAll
    from dice_embeddings_b200.ops import kernels
    from dice_embeddings_b200.ops.hybrid_step import ExternalQueryEngine
    gen = _gen(seed)
    ds = KvsAll(_graph(case, seed), case["entities"], case["relations"], label_smoothing_rate=0.1).to(DEV)
    name, extra = case["model"], dict(num_of_output_channels=case["channels"], kernel_size=3)
    if name == "Keci12":
        name, extra = "Keci", {}
    torch.manual_seed(seed % (2 ** 31))
    model = _model(name, case, "Adam", "KvsAll", **extra) if case["model"] != "Keci12" else _keci12(case)
    model.train()
    with torch.no_grad():
        for p_name, prm in model.named_parameters():
            if "embeddings" in p_name:
                _load(prm, gen, 0.25)
            elif "coefficients" in p_name:
                prm.fill_(0.7)
    init = {k: v.detach().clone() for k, v in model.state_dict().items()}
    engine = ExternalQueryEngine(model, ds, batch_size=case["batch"], lr=0.001, device=DEV)
    idx = torch.randperm(len(ds), device=DEV, generator=gen)[:case["batch"]]
    batch = ds.make_batch(idx)
    for _ in range(2):
        engine.step(batch)
    with torch.no_grad():
        model.load_state_dict(init)
        kernels.cast_bf16(engine.E, engine.E_bf16)
        g_ent = 0.1 / (math.sqrt(case["batch"]) * case["entities"])
        _load_moments(engine.mE, engine.vE, gen, g_ent)
        engine.step_count.fill_(200)
        if engine.rest_optimizer is not None:
            for st in engine.rest_optimizer.state.values():
                st["exp_avg"].zero_()
                st["exp_avg_sq"].fill_((10 * g_ent) ** 2)
                st["step"].fill_(200.0)
    return dict(engine=engine, batch=batch, model=model)


def _keci12(case):
    from dice_embeddings_b200.models import initialize_model
    with torch.device(DEV):
        return initialize_model(dict(model="Keci", embedding_dim=case["dim"], num_entities=case["entities"],
                                     num_relations=case["relations"], optim="Adam", learning_rate=0.01,
                                     scoring_technique="KvsAll", p=1, q=2))[0]


def _positives(case, gen):
    ne, n = case["entities"], case["batch"]
    e = (ne * torch.rand(n, 2, device=DEV, generator=gen) ** 3).long().clamp_(max=ne - 1)   # heavy-tailed ids
    r = torch.randint(0, case["relations"], (n,), device=DEV, generator=gen)
    return torch.stack((e[:, 0], r, e[:, 1]), dim=1).contiguous()


def _prepare_sampled(case, seed):
    from dice_embeddings_b200.ops.sampled_step import FusedSampledEngine
    gen = _gen(seed)
    model = _model(case["model"], case, case["optim"], case["technique"])
    engine = FusedSampledEngine(model, case["technique"], lr=0.01, device=DEV, neg_ratio=case["negatives"],
                                label_smoothing=0.1, seed=seed % (2 ** 31))
    pos = _positives(case, gen)
    if case["technique"] == "NegSample":
        batch = (pos,)
    else:
        C = 1 + case["negatives"]
        cand = torch.randint(0, case["entities"], (pos.shape[0], C), device=DEV, generator=gen)
        cand[:, 0] = pos[:, 2]
        labels = torch.zeros(pos.shape[0], C, device=DEV)
        labels[:, 0] = 1.0
        if case["technique"] == "KvsSample":   # the first columns of a row are its known tails
            known = 1 + (4 * torch.rand(pos.shape[0], 1, device=DEV, generator=gen) ** 2).long()
            labels = (torch.arange(C, device=DEV).unsqueeze(0) < known).float()
        batch = (pos[:, :2].contiguous(), cand, labels)
    engine.step(batch)
    pairs = case["batch"] * (1 + case["negatives"])
    _resume(engine, case, gen, 0.2 / pairs, 2.0 / pairs)
    return dict(engine=engine, batch=batch)


def _prepare_rowsparse(case, seed):
    import torch.distributed as dist
    from dice_embeddings_b200.parallel.sharded_sampled import ShardedSampledEngine
    if not dist.is_initialized():   # one rank: the process group of the sharded trainer
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device(DEV))
    gen = _gen(seed)
    small = dict(case, entities=8)   # relation table and hyper-parameters; the entity rows live in the engine
    model = _model(case["model"], small, "Adam", "NegSample")
    model.num_entities = case["entities"]
    rows = torch.empty(case["entities"], case["dim"], device=DEV)
    _load(rows, gen, 0.25)
    engine = ShardedSampledEngine(model, "NegSample", batch_size=case["batch"], lr=0.01, neg_ratio=case["negatives"],
                                  label_smoothing=0.1, device=DEV, layout="tails", entity_rows=rows,
                                  seed=seed % (2 ** 31))
    batch = (_positives(case, gen),)
    for _ in range(2):
        engine.step(batch)
    pairs = case["batch"] * (1 + case["negatives"])
    _resume(engine, case, gen, 0.2 / pairs, 2.0 / pairs)
    return dict(engine=engine, batch=batch)


@torch.no_grad()
def _prepare_evaluate(case, seed):
    from dice_embeddings_b200.data.vocab import er_csr
    gen = _gen(seed)
    triples = _graph(case, seed)
    rng = np.random.default_rng(seed + 1)
    test = triples[rng.permutation(len(triples))[:case["queries"]]]
    model = _model(case["model"], case, "Adam", "KvsAll").eval()
    _load(model.entity_embeddings.weight, gen, 0.25)
    _load(model.relation_embeddings.weight, gen, 1.0)
    # the tails lean towards the query vectors of their triples, as they do in a trained model
    t = torch.from_numpy(test).to(DEV)
    q, _ = model.compose(*model.get_head_relation_representation(t[:, :2]))
    lean = torch.zeros_like(model.entity_embeddings.weight).index_put_((t[:, 2],), q, accumulate=True)
    deg = torch.zeros(case["entities"], device=DEV).index_add_(0, t[:, 2], torch.ones_like(t[:, 2], dtype=torch.float32))
    strength = 4.0 * torch.rand(case["entities"], 1, device=DEV, generator=gen) / math.sqrt(case["dim"])
    model.entity_embeddings.weight.add_(strength * lean / deg.clamp_min(1.0).sqrt().unsqueeze(1))
    return dict(model=model, test=test, er=er_csr(triples, case["relations"]), batch=case["batch"])


@torch.no_grad()
def _prepare_table(case, seed):
    from dice_embeddings_b200.ops.eval_rank import FusedRanker
    gen = _gen(seed)
    ne, d, n = case["entities"], case["dim"], case["queries"]
    table = torch.randn(ne, d, device=DEV, generator=gen).mul_(0.25)
    q = torch.randn(n, d, device=DEV, generator=gen).mul_(0.25)
    # every query has one entity that scores two to five standard deviations above the rest, as in a trained model
    tgt = torch.randperm(ne, device=DEV, generator=gen)[:n]
    lift = (2.0 + 3.0 * torch.rand(n, 1, device=DEV, generator=gen)) / math.sqrt(d)
    table[tgt] = 0.3 * table[tgt] + lift * q
    state = dict(ranker=FusedRanker(table.to(torch.bfloat16)), q=q)
    if case["kind"] == "topk":
        state["k"] = case["k"]
        return state
    F = case["filters"]
    cols = (ne * torch.rand(n, F, device=DEV, generator=gen) ** 3).long().clamp_(max=ne - 1).to(torch.int32)
    cols[:, 0] = tgt.to(torch.int32)
    state.update(target=tgt, ptr=torch.arange(n + 1, device=DEV) * F, cols=cols.reshape(-1))
    return state


def prepare(case, seed):
    kind = case["kind"]
    make = dict(kvsall=_prepare_kvsall, hybrid=_prepare_hybrid, sampled=_prepare_sampled,
                rowsparse=_prepare_rowsparse, evaluate=_prepare_evaluate, rank=_prepare_table, topk=_prepare_table)
    return dict(make[kind](case, seed), kind=kind)


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "evaluate":
        from dice_embeddings_b200.evaluation.ranking import tail_ranks
        return tail_ranks(state["model"], state["test"], state["er"], state["batch"])
    if kind == "rank":
        return state["ranker"].ranks(state["q"], state["target"], state["ptr"], state["cols"])
    if kind == "topk":
        return state["ranker"].topk(state["q"], state["k"])
    e = state["engine"]
    out = dict(loss=e.step(state["batch"]), E=e.E, mE=e.mE)
    if kind == "hybrid":
        out.update({n: p for n, p in state["model"].named_parameters() if not n.startswith("entity_embeddings")})
    else:
        out.update(R=e.R, mR=e.mR)
        if e.coeff is not None:
            out["coeff"] = e.coeff
    return out


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    kind, ne, d = case["kind"], case["entities"], case["dim"]
    if kind in ("kvsall", "hybrid", "sampled"):
        table = 2 * 3 * 4 * ne * d                               # weights and two moments, read and written once
        if kind == "sampled":
            n = case["batch"] * (1 + case["negatives"])
            return dict(bytes=table + 4 * n * d + 8 * n, flops=6 * n * d)
        n = case["batch"]
        conv = 0
        if kind == "hybrid" and case["model"] in ("ConEx", "AConEx", "ConvQ"):
            c = case["channels"]
            conv = 3 * n * (2 * d * c * 18 + 2 * (2 * d * c) * d * (2 if case["model"] == "AConEx" else 1))
        return dict(bytes=table + 4 * n * d, flops=6 * n * ne * d + conv)
    if kind == "rowsparse":
        n = case["batch"] * (1 + case["negatives"])
        touched = ne * -math.expm1(-n / ne)                      # expected number of distinct rows
        return dict(bytes=4 * d * (6 * touched + n) + 8 * n, flops=6 * n * d)
    n = case["queries"]
    if kind == "evaluate":
        return dict(bytes=4 * ne * d + 4 * n * d, flops=2 * n * ne * d)
    return dict(bytes=2 * ne * d + 4 * n * d, flops=2 * n * ne * d)


def tolerance(case):
    kind = case["kind"]
    # Four times what the same step shows against 64-bit arithmetic on the same inputs.
    if kind in ("kvsall", "hybrid"):
        # bf16 operands and bf16 logit gradients: rel 2.4e-3 on the gradients, single entries of rows with few
        # contributions up to 0.08
        return {"rel": 1e-2, "max": 0.3}
    if kind in ("sampled", "rowsparse"):
        return {"rel": 2e-6, "max": 4e-5}     # fp32 throughout: rel 4.9e-7 on the gradients, 9e-6 on single entries
    # 32-bit sums in another order: scores to about 2e-6, a rank moves where two scores are that close
    return {"rel": 1e-5, "max": 1e-4, "differ": 2e-3}
