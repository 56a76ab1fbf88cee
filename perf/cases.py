"""What this framework is timed on: the steps that a training or scoring program has it do, through its public calls.

Every case is one of seven kinds of work, ``case["kind"]``:

    deepfm      one DeepFM training step (models.DeepFM + bce_with_logits + Optimizer.step), or a scoring pass
    multihot    one training step of the multi-hot Wide&Deep model: bags of ids in a combined table
    wide_deep   one training step of the single-hot Wide&Deep model
    mlp         one training step of a dense MLP, with or without compressed (DCT) gradients
    pull_push   one sparse table: apply a step's gradients, then fetch the rows again
    combine     many small tables through the combined calls: apply gradients, fetch rows
    bags        an embedding-bag layer (JaggedEmbedding), forward and backward

``draw`` spreads the same kinds over the sizes, widths, optimizers and options that their callers use.  A state is one
job: an engine with tables as a job some hours in would hold them (rows and optimizer state are imported), the model,
and one batch.  ``exact`` computes what the first pass on such a state returns in float64 with plain torch.
"""
import math

import torch

import kraken_b200.pytorch as kk
from kraken_b200.models import MLP, DeepFM, MultiHotWideAndDeep, WideAndDeep
from kraken_b200.ops import bce_with_logits
from kraken_b200.pytorch import native
from kraken_b200.utils.graph import GraphedStep

_NUM_DENSE = 13
_OPTIMS = ("sgd", "momentum", "adagrad", "adam", "amsgrad", "rmsprop")


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # The benchmark's step on one GPU: global batch 65536, ids over 26 x 1e7, captured as a CUDA graph.
        _deepfm("deepfm_step_b65536", 65536, vocab=10_000_000, graph=True, fold=True, slots_log2=25),
        # The same step at the share of one of eight GPUs.
        _deepfm("deepfm_step_b8192", 8192, vocab=10_000_000, graph=True, fold=True, slots_log2=25),
        # examples/deepfm/main.py as it stands: batch 4096, vocabulary 1e5, two tables, launched from Python.
        _deepfm("deepfm_script_b4096", 4096, vocab=100_000, graph=False, fold=False),
        # Scoring a held-out set with the trained model; its last batch is a ragged one.
        _deepfm("deepfm_score_b1789", 1789, vocab=100_000, graph=False, fold=False, train=False),
        # Multi-hot Wide&Deep, a quarter of the benchmark's 16384 samples per GPU: 8 million ids, Adagrad.
        {"name": "multihot_step_b4096", "kind": "multihot", "batch": 4096, "fields": 100, "vocab": (1 << 40) // 100,
         "zipf": 1.1, "mean_len": 20, "dim": 64, "hidden": "1024-512-256", "optim": "adagrad"},
        # Single-hot Wide&Deep at the batch of the CPU configuration: the smallest training step.
        {"name": "wide_deep_step_b512", "kind": "wide_deep", "batch": 512, "fields": 26, "vocab": 100_000,
         "zipf": 1.05, "dim": 8, "hidden": "256-128", "optim": "adagrad"},
        # The dense-table path: MLP 784-4096-4096-4096-10, batch 1024, SGD with momentum, as a CUDA graph ...
        {"name": "mlp_step_b1024", "kind": "mlp", "batch": 1024, "hidden": "4096-4096-4096", "classes": 10,
         "optim": "momentum", "graph": True, "dct": False},
        # ... and with DCT gradient compression (its threshold refresh keeps it out of a graph).
        {"name": "mlp_dct_step_b1024", "kind": "mlp", "batch": 1024, "hidden": "4096-4096-4096", "classes": 10,
         "optim": "momentum", "graph": False, "dct": True},
        # The huge-table configuration: 131072 samples x 26 ids, Zipf(0.9) over 1e9, dim 64, Adagrad.
        {"name": "pull_push_3407872x64", "kind": "pull_push", "n": 131072 * 26, "dim": 64, "space": 1_000_000_000,
         "zipf": 0.9, "optim": "adagrad"},
        # A small odd-width table: ids of one field of a small job, row width not a multiple of 4.
        {"name": "pull_push_5003x10", "kind": "pull_push", "n": 5003, "dim": 10, "space": 100_000, "zipf": 1.1,
         "optim": "adam"},
        # The reference's DeepFM layout, a dim-1 and a dim-4 table for each of 39 fields, in one combined call.
        {"name": "combine_39x2_b4096", "kind": "combine", "fields": 39, "batch": 4096, "dim": 4, "vocab": 1_000_000,
         "zipf": 1.1, "optim": "adam"},
        # An EmbeddingBag layer by itself: ragged weighted bags, some of them empty, mean pooling.
        {"name": "bags_20011x24_mean", "kind": "bags", "bags": 20011, "mean_len": 12, "dim": 24, "space": 5_000_000,
         "zipf": 1.05, "mode": "mean", "weights": True, "optim": "adagrad"},
    ]


def _deepfm(name, batch, vocab, graph, fold, train=True, slots_log2=0, fields=26, dim=16, hidden="400-400-400",
            optim="adam"):
    c = {"kind": "deepfm", "batch": batch, "fields": fields, "vocab": vocab, "zipf": 1.1, "dim": dim, "hidden": hidden,
         "optim": optim, "fold": fold, "graph": graph, "train": train, "slots_log2": slots_log2}
    return dict(c, name=name) if name else c


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("deepfm", "deepfm", "deepfm", "multihot", "wide_deep", "mlp", "pull_push", "pull_push",
                       "combine", "bags"))
    optim = rng.choice(_OPTIMS)
    if kind == "deepfm":
        train = rng.random() < 0.75
        return _deepfm(None, _log_int(rng, 200, 65536), vocab=_log_int(rng, 10_000, 10_000_000),
                       graph=train and rng.random() < 0.6, fold=rng.random() < 0.5, train=train,
                       fields=rng.randint(8, 39), dim=rng.choice((8, 16, 16, 32)),
                       hidden=rng.choice(("400-400-400", "256-128", "512-256-64")), optim=optim)
    if kind == "multihot":
        fields, mean_len = rng.randint(10, 100), rng.randint(3, 25)
        most = min(4096, 8_000_000 // (fields * mean_len))
        return {"kind": kind, "batch": _log_int(rng, 64, most), "fields": fields,
                "vocab": _log_int(rng, 100_000, (1 << 40) // 100), "zipf": round(rng.uniform(1.02, 1.2), 3),
                "mean_len": mean_len, "dim": rng.choice((16, 32, 64)),
                "hidden": rng.choice(("1024-512-256", "256-128")), "optim": optim}
    if kind == "wide_deep":
        return {"kind": kind, "batch": _log_int(rng, 100, 16384), "fields": rng.randint(8, 39),
                "vocab": _log_int(rng, 1000, 1_000_000), "zipf": round(rng.uniform(1.02, 1.2), 3),
                "dim": rng.choice((4, 8, 16)), "hidden": rng.choice(("256-128", "128-64")), "optim": optim}
    if kind == "mlp":
        dct = rng.random() < 0.4
        widths = rng.choice(("4096-4096-4096", "2048-2048", "1024-512", "512-512-256"))
        return {"kind": kind, "batch": _log_int(rng, 100, 1024), "hidden": widths, "classes": rng.choice((1, 10, 16)),
                "optim": optim, "graph": not dct and rng.random() < 0.5, "dct": dct}
    if kind == "pull_push":
        dim = rng.choice((1, 4, 8, 10, 16, 32, 64, 64, 100, 128))
        return {"kind": kind, "n": _log_int(rng, 300, min(3_400_000, 200_000_000 // dim)), "dim": dim,
                "space": _log_int(rng, 10_000, 1_000_000_000), "zipf": round(rng.uniform(0.85, 1.2), 3), "optim": optim}
    if kind == "combine":
        return {"kind": kind, "fields": rng.randint(3, 39), "batch": _log_int(rng, 64, 8192),
                "dim": rng.choice((4, 8, 10, 16)), "vocab": _log_int(rng, 1000, 1_000_000),
                "zipf": round(rng.uniform(1.02, 1.2), 3), "optim": optim}
    return {"kind": kind, "bags": _log_int(rng, 100, 100_000), "mean_len": rng.randint(1, 30),
            "dim": rng.choice((8, 17, 24, 32, 64)), "space": _log_int(rng, 10_000, 10_000_000),
            "zipf": round(rng.uniform(0.95, 1.2), 3), "mode": rng.choice(("sum", "mean")),
            "weights": rng.random() < 0.5, "optim": optim}


# ---------------------------------------------------------------------------------------------- inputs
def _optim(name):
    return {"sgd": kk.SGD(), "momentum": kk.SGD(momentum=0.9), "adagrad": kk.Adagrad(initial_accumulator_value=0.1),
            "adam": kk.Adam(), "amsgrad": kk.Adam(amsgrad=True), "rmsprop": kk.RMSprop()}[name]


_LR = {"sgd": 0.05, "momentum": 0.05, "adagrad": 0.01, "adam": 1e-3, "amsgrad": 1e-3, "rmsprop": 1e-3}
_STEPS = 100  # updates that rows and weights have seen before the timed one
# checkpoint state types (kraken/protocol names): momentum buffer, state sum, first / second moment, its maximum, square average
_MOMENTUM, _STATE_SUM, _FIRST, _SECOND, _SECOND_MAX, _SQUARE = 1, 2, 3, 4, 5, 6


class _Draw:
    """Seeded random inputs on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev).manual_seed(int(seed) * 2 + 1)

    def normal(self, shape, std=1.0):
        return torch.randn(shape, generator=self.gen, device=self.dev) * std

    def uniform(self, shape, lo, hi):
        return torch.rand(shape, generator=self.gen, device=self.dev) * (hi - lo) + lo

    def zipf(self, shape, vocab, s):
        """Ranks in [0, vocab) with P(r) ~ (r + 1)^-s."""
        u = torch.rand(shape, generator=self.gen, device=self.dev, dtype=torch.float64)
        a = 1.0 - s if s != 1.0 else 1e-6
        r = ((float(vocab + 1) ** a - 1.0) * u + 1.0) ** (1.0 / a) - 1.0
        return r.long().clamp_(0, vocab - 1)

    def state(self, optim, shape, grad_std):
        """Optimizer state after some updates with gradients of about ``grad_std``."""
        g2 = grad_std * grad_std
        if optim == "momentum":
            return {_MOMENTUM: self.normal(shape, 2 * grad_std)}
        if optim == "adagrad":
            return {_STATE_SUM: self.uniform(shape, 0.1, 0.1 + 50 * g2)}
        if optim in ("adam", "amsgrad"):
            s = {_FIRST: self.normal(shape, 0.3 * grad_std), _SECOND: self.uniform(shape, 0.05 * g2, 0.2 * g2)}
            if optim == "amsgrad":
                s[_SECOND_MAX] = self.uniform(shape, 0.5 * g2, 2 * g2)
            return s
        if optim == "rmsprop":
            return {_SQUARE: self.uniform(shape, 0.5 * g2, 2 * g2)}
        return {}

    def rows(self, ids, dim, optim, std, grad_std):
        """Table contents for ``ids``, as a checkpoint would hold them."""
        n = ids.numel()
        steps = {0: torch.full((n,), _STEPS, dtype=torch.int64, device=self.dev)} if _counts(optim) else {}
        return {"dim": dim, "ids": ids, "vals": self.normal((n, dim), std),
                "states": self.state(optim, (n, dim), grad_std), "states_i": steps}

    def weights(self, sizes, optim):
        """[(name suffix, checkpoint value)] of an MLP with layers sizes[0] -> sizes[1] -> ..."""
        out = []
        for i, (k, n) in enumerate(zip(sizes[:-1], sizes[1:])):
            bound = 1.0 / math.sqrt(k)
            for part, shape in (("weight", (n, k)), ("bias", (n,))):
                out.append((f"layers.{i}.{part}", self.dense(self.uniform(shape, -bound, bound), optim)))
        return out

    def dense(self, val, optim):
        return {"val": val, "states": self.state(optim, tuple(val.shape), 1e-3),
                "states_i": {0: _STEPS} if _counts(optim) else {}}


def _counts(optim):
    return optim in ("momentum", "adam", "amsgrad")


def _hidden(case):
    return [int(x) for x in case["hidden"].split("-")]


def _pad8(width):
    return (width + 7) // 8 * 8


def _hash40(x):
    """The 2^40 id space of the combined table: an invertible mix of (field, rank), truncated."""
    x = x ^ (x >> 29)
    x = x * 0x1E35A7BD2B1D6F53
    x = x ^ ((x >> 32) & 0xFFFFFFFF)
    return x & ((1 << 40) - 1)


def _field_ids(r, case, batch):
    F, vocab = case["fields"], case["vocab"]
    return r.zipf((batch, F), vocab, case["zipf"]) + torch.arange(F, device=r.dev) * vocab


def _click(r, case):
    dense = torch.log1p(torch.exp(r.normal((case["batch"], _NUM_DENSE))))
    labels = (r.uniform((case["batch"],), 0.0, 1.0) < 0.3).float()
    return dense, labels


def _lens(r, bags, mean_len, lowest):
    """Bag lengths ~ Poisson(mean_len) clipped to [lowest, 100]."""
    rate = torch.full((bags,), float(mean_len), device=r.dev)
    lens = torch.poisson(rate, generator=r.gen).long().clamp_(lowest, 100)
    off = torch.zeros(bags + 1, dtype=torch.int64, device=r.dev)
    torch.cumsum(lens, 0, out=off[1:])
    return lens, off


def _inputs(case, seed):
    """Everything a case starts from: the batch, the tables' rows, the dense weights."""
    r = _Draw(seed)
    kind, optim = case["kind"], case["optim"]
    d = {"tables": {}, "weights": []}
    if kind == "deepfm":
        B, F, dim = case["batch"], case["fields"], case["dim"]
        d["dense"], d["labels"] = _click(r, case)
        d["ids"] = _field_ids(r, case, B)
        d["earlier"] = _field_ids(r, case, B)   # an earlier batch: rows that exist, ids a warm-up uses
        # one id in fifty that the earlier batch did not hold is new to the table, as on a day's new items
        here = torch.unique(d["ids"])
        new = ~torch.isin(here, d["earlier"]) & (r.uniform(tuple(here.shape), 0.0, 1.0) < 0.02)
        known = torch.unique(torch.cat([here[~new], d["earlier"].reshape(-1)]))
        g = 0.3 / B
        if case["fold"]:
            row = (dim + 4) // 4 * 4
            d["tables"]["embedding_and_first_order"] = r.rows(known, row, optim, 0.05, g)
        else:
            d["tables"]["first_order"] = r.rows(known, 1, optim, 0.05, g)
            d["tables"]["second_order"] = r.rows(known, dim, optim, 0.05, g)
        d["sizes"] = [_pad8(F * dim + _NUM_DENSE)] + _hidden(case) + [1]
        d["weights"] = [("mlp." + k, v) for k, v in r.weights(d["sizes"], optim)]
    elif kind in ("wide_deep", "multihot"):
        B, F, dim = case["batch"], case["fields"], case["dim"]
        d["dense"], d["labels"] = _click(r, case)
        if kind == "wide_deep":
            d["ids"] = _field_ids(r, case, B)
        else:
            lens, d["offsets"] = _lens(r, B * F, case["mean_len"], 1)
            field = torch.arange(F, device=r.dev).repeat(B).repeat_interleave(lens)
            d["ids"] = _hash40(r.zipf(tuple(field.shape), case["vocab"], case["zipf"]) + field * case["vocab"])
        known = torch.unique(d["ids"])
        d["tables"]["wide"] = r.rows(known, 1, optim, 0.05, 0.3 / B)
        d["tables"]["deep" if kind == "wide_deep" else "combined"] = r.rows(known, dim, optim, 0.05, 0.3 / B)
        d["sizes"] = [_pad8(F * dim + _NUM_DENSE)] + _hidden(case) + [1]
        d["weights"] = [("bias", r.dense(r.normal((1,), 0.1), optim))]
        d["weights"] += [("mlp." + k, v) for k, v in r.weights(d["sizes"], optim)]
    elif kind == "mlp":
        B, C = case["batch"], case["classes"]
        means = r.normal((max(C, 2), 784))
        d["labels"] = (r.uniform((B,), 0.0, 1.0) * max(C, 2)).long().clamp_(0, max(C, 2) - 1)
        d["dense"] = means[d["labels"]] + r.normal((B, 784))
        d["sizes"] = [784] + _hidden(case) + [C]
        d["weights"] = r.weights(d["sizes"], optim)
    elif kind == "pull_push":
        d["ids"] = r.zipf((case["n"],), case["space"], case["zipf"])
        d["grads"] = r.normal((case["n"], case["dim"]), 0.01)
        d["tables"]["table"] = r.rows(torch.unique(d["ids"]), case["dim"], optim, 0.05, 0.01)
    elif kind == "combine":
        d["ids"], d["grads"] = [], []
        for w, dim in ((0, 1), (1, case["dim"])):
            for f in range(case["fields"]):
                ids = r.zipf((case["batch"],), case["vocab"], case["zipf"]) if w == 0 else d["ids"][f]
                d["ids"].append(ids)
                d["grads"].append(r.normal((case["batch"], dim), 0.01))
                d["tables"][f"t{w}.{f}"] = r.rows(torch.unique(ids), dim, optim, 0.05, 0.01)
    else:
        lens, d["offsets"] = _lens(r, case["bags"], case["mean_len"], 0)
        n = int(d["offsets"][-1])
        d["ids"] = r.zipf((n,), case["space"], case["zipf"])
        d["bag_weights"] = r.uniform((n,), 0.1, 2.0) if case["weights"] else None
        d["grads"] = r.normal((case["bags"], case["dim"]), 0.01)
        d["tables"]["bag"] = r.rows(torch.unique(d["ids"]), case["dim"], optim, 0.05, 0.01)
    return d


# ---------------------------------------------------------------------------------------------- states
class _Job:
    """One training job.  A process runs one at a time, so a job takes its engine's place before each pass."""

    def __init__(self, **options):
        native._engine = None
        kk.initialize("gpu", **options)
        self.engine = native.engine()

    def enter(self):
        native._engine = self.engine

    def load(self, d, prefix):
        """Puts rows, weights and optimizer state in place, as loading a checkpoint does."""
        for name, value in d["weights"]:
            self.engine.import_dense(self.engine.name_to_id[name], name, value)
        for name, cols in d["tables"].items():
            self.engine.import_sparse(self.engine.name_to_id[prefix + name], cols)


def _slots(d, case):
    rows = max([int(t["ids"].numel()) for t in d["tables"].values()], default=1)
    return max(1 << case.get("slots_log2", 0), 1 << max(14, (3 * rows).bit_length()))


def prepare(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    options = {"table_capacity": _slots(d, case), "seed": 0}
    if kind == "deepfm":
        options.update(max_ids_per_call=case["batch"] * case["fields"], overlap_dense_step=case["graph"])
    elif kind == "multihot":
        most = int(case["batch"] * case["fields"] * (case["mean_len"] + 1) * 1.05) + 4096
        options.update(max_ids_per_call=most, max_unique_per_call=max(1 << 20, most // 2))
    elif kind == "mlp":
        options.update(overlap_dense_step=case["graph"],
                       emitter_type=kk.EmitterType.kDCT if case["dct"] else kk.EmitterType.kDefault)
    job = _Job(**options)
    dev = job.engine.device
    state = {"case": case, "job": job}
    torch.manual_seed(int(seed))

    if kind in ("pull_push", "combine"):
        o = _optim(case["optim"])
        kk.init_model("tables", o.type(), o.conf())
        kk.update_lr(_LR[case["optim"]])
        tids = [kk.register_sparse_table(name, t["dim"], torch.float32, kk.InitializerType.kConstant, {"value": "0.0"})
                for name, t in d["tables"].items()]
        job.load(d, "")
        state.update(tids=tids, ids=d["ids"], grads=d["grads"])
        return state
    if kind == "bags":
        layer = kk.JaggedEmbedding(case["dim"], initializer=kk.ConstantInitializer(0.0), name="bag", mode=case["mode"],
                                   patch_value=0.25)
        kk.Optimizer("bags", layer.named_parameters(), _LR[case["optim"]], _optim(case["optim"]))
        job.load(d, "")
        state.update(layer=layer, grads=d["grads"],
                     bags=kk.JaggedTensor(d["ids"], d["offsets"], d["bag_weights"], validate=False))
        return state

    if kind == "deepfm":
        model = DeepFM(case["fields"], _NUM_DENSE, case["dim"], _hidden(case), init_std=0.0,
                       fold_first_order=case["fold"]).to(dev)
        prefix, batch = "deepfm.", (d["dense"], d["ids"], d["labels"])
    elif kind == "wide_deep":
        model = WideAndDeep(case["fields"], _NUM_DENSE, case["dim"], _hidden(case)).to(dev)
        prefix, batch = "wide_deep.", (d["dense"], d["ids"], d["labels"])
    elif kind == "multihot":
        model = MultiHotWideAndDeep(case["fields"], _NUM_DENSE, case["dim"], _hidden(case),
                                    mean_fields=range(0, case["fields"], 2)).to(dev)
        prefix, batch = "mh_wide_deep.", (d["dense"], d["ids"], d["offsets"], d["labels"])
    else:
        model = MLP(784, _hidden(case) + [case["classes"]]).to(dev)
        prefix, batch = "", (d["dense"], d["labels"])
    opt = kk.Optimizer("model", model.named_parameters(), _LR[case["optim"]], _optim(case["optim"]))

    def step(*inputs):
        if kind == "multihot":
            dense, ids, offsets, labels = inputs
            logits = model(dense, kk.JaggedTensor(ids, offsets, validate=False))
        else:
            labels, logits = inputs[-1], model(*inputs[:-1])
        if kind != "mlp":
            loss = bce_with_logits(logits, labels)
        elif case["classes"] > 1:
            loss = torch.nn.functional.cross_entropy(logits, labels)
        else:
            loss = bce_with_logits(logits.squeeze(-1), labels.float())
        loss.backward()
        opt.step()
        return loss.detach(), logits.detach()

    state.update(model=model, step=step, batch=batch)
    if case.get("graph"):
        job.load(d, prefix)
        warm = (d["dense"], d["earlier"], d["labels"]) if kind == "deepfm" else batch
        state["step"] = GraphedStep(step, warm, warmup=2, optimizer=opt)
    job.load(d, prefix)  # after the warm-up steps: the state that the first timed pass starts from
    if case.get("train", True):
        # The weights are views of the engine's memory: whoever holds a pass's outputs keeps the job.
        params = dict(model.named_parameters())
        state["weights"] = {}
        for name, _ in d["weights"]:
            view = params[name].detach()
            view.job = job
            state["weights"][name] = view
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    state["job"].enter()
    if kind == "pull_push":
        kk.push_sparse_table(state["tids"][0], state["ids"], state["grads"])
        return kk.pull_sparse_table(state["tids"][0], state["ids"])
    if kind == "combine":
        kk.combine_push_sparse_table(state["tids"], state["ids"], state["grads"])
        return kk.combine_pull_sparse_table(state["tids"], state["ids"])[::2]  # 64 outputs at most are compared
    if kind == "bags":
        out = state["layer"](state["bags"])
        out.backward(state["grads"])
        return out.detach()
    if not case.get("train", True):
        with torch.no_grad():
            return state["model"](*state["batch"][:-1])
    loss, logits = state["step"](*state["batch"])
    return {"loss": loss, "logits": logits, "weights": state["weights"]}


# ---------------------------------------------------------------------------------------------- the floor
def _distinct(n, vocab, s):
    """Expected number of distinct ids among n draws of the Zipf envelope over ``vocab`` ranks."""
    a, total, lo = (1.0 - s if s != 1.0 else 1e-6), 0.0, 1.0
    cdf = (lambda x: (x ** a - 1.0) / (float(vocab + 1) ** a - 1.0))
    while lo < vocab + 1:
        hi = min(float(vocab + 1), max(lo + 1.0, lo * 1.02))
        count, mass = hi - lo, cdf(hi) - cdf(lo)
        total += count * -math.expm1(-n * mass / count) if n * mass / count < 700 else count
        lo = hi
    return total


_SLABS = {"sgd": 0, "momentum": 1, "adagrad": 1, "adam": 2, "amsgrad": 3, "rmsprop": 1}


def _row_update(u, dim, optim):
    """Bytes of updating u rows: key, value and state slabs read and written, the step counter."""
    return u * (8 + 8 * dim * (1 + _SLABS[optim]) + (8 if _counts(optim) else 0))


def work(case):
    kind, optim = case["kind"], case["optim"]
    if kind == "pull_push":
        n, dim = case["n"], case["dim"]
        u = _distinct(n, case["space"], case["zipf"])
        return {"bytes": 8 * n + 8 * n * dim + _row_update(u, dim, optim), "flops": n * dim}
    if kind == "combine":
        n, F = case["batch"], case["fields"]
        u = _distinct(n, case["vocab"], case["zipf"])
        return {"bytes": F * sum(8 * n + 8 * n * dim + _row_update(u, dim, optim) for dim in (1, case["dim"])),
                "flops": F * n * (1 + case["dim"])}
    if kind == "bags":
        k, dim = case["bags"], case["dim"]
        n = k * case["mean_len"]
        u = _distinct(n, case["space"], case["zipf"])
        return {"bytes": n * (12 if case["weights"] else 8) + 8 * k + 8 * k * dim + _row_update(u, dim, optim),
                "flops": 4 * n * dim}
    B = case["batch"]
    inputs = 784 if kind == "mlp" else _pad8(case["fields"] * case["dim"] + _NUM_DENSE)
    sizes = [inputs] + _hidden(case) + [case.get("classes", 1)]
    params = sum(k * n + n for k, n in zip(sizes[:-1], sizes[1:]))
    macs = B * sum(k * n for k, n in zip(sizes[:-1], sizes[1:]))
    train = case.get("train", True)
    flops = 2 * macs * (3 if train else 1)
    if kind == "mlp":
        flops -= 2 * B * sizes[0] * sizes[1]  # no gradient of the images
        dct = 8 * params if case["dct"] else 0  # the residual that is carried along
        return {"bytes": 4 * B * 784 + 8 * params * (1 + _SLABS[optim]) + dct, "flops": flops}
    F = case["fields"]
    per_field = B * (case["mean_len"] if kind == "multihot" else 1)
    n = per_field * F
    u = F * _distinct(per_field, case["vocab"], case["zipf"])
    width = case["dim"] + 1
    data = 8 * n + 4 * B * (_NUM_DENSE + 2) + (8 * B * F if kind == "multihot" else 0)
    if not train:
        return {"bytes": data + 4 * params + u * (8 + 4 * width), "flops": flops + 3 * n * case["dim"]}
    return {"bytes": data + 8 * params * (1 + _SLABS[optim]) + _row_update(u, width, optim),
            "flops": flops + 6 * n * case["dim"]}


# ---------------------------------------------------------------------------------------------- correctness
def tolerance(case):
    kind = case["kind"]
    if kind in ("pull_push", "combine", "bags"):
        return {"rel": 1e-5, "max": 1e-3}   # float32 sums in any order
    # bf16 operands in the MLP; an optimizer that divides by a small second moment amplifies it in the weights
    return {"rel": 1e-2, "max": 0.2}


def _update64(optim, lr, g, w, states, steps):
    """One server-side update in float64; returns the new value."""
    s = {k: v.double() for k, v in states.items()}
    if optim == "sgd":
        return w - lr * g
    if optim == "momentum":
        return w - lr * (0.9 * s[_MOMENTUM] + g)
    if optim == "adagrad":
        return w - lr * g / ((s[_STATE_SUM] + g * g).sqrt() + 1e-10)
    if optim == "rmsprop":
        return w - lr * g / ((0.99 * s[_SQUARE] + 0.01 * g * g).sqrt() + 1e-8)
    t = steps + 1
    m = (0.9 * s[_FIRST] + 0.1 * g) / (1 - 0.9 ** t)
    v = (0.999 * s[_SECOND] + 0.001 * g * g) / (1 - 0.999 ** t)
    if optim == "amsgrad":
        v = torch.maximum(v, s[_SECOND_MAX])
    return w - lr * m / (v.sqrt() + 1e-8)


def _rows64(table, ids):
    """Rows of ids in float64; an id that the table does not hold gives zeros, the initial value."""
    at = torch.searchsorted(table["ids"], ids.reshape(-1)).clamp_(max=table["ids"].numel() - 1)
    rows = table["vals"][at].double()
    rows[table["ids"][at] != ids.reshape(-1)] = 0
    return rows.view(*ids.shape, table["dim"])


def _pushed64(table, ids, grads, optim):
    """What a pull returns after the push of grads: every id's rows, updated with the sum of its gradients."""
    at = torch.searchsorted(table["ids"], ids)
    g = torch.zeros(table["vals"].shape, dtype=torch.float64, device=ids.device).index_add_(0, at, grads.double())
    return _update64(optim, _LR[optim], g, table["vals"].double(), table["states"], _STEPS)[at]


def _pool64(table, ids, offsets, weights=None):
    at = torch.searchsorted(table["ids"], ids)
    return torch.nn.functional.embedding_bag(at, table["vals"].double(), offsets, mode="sum", include_last_offset=True,
                                             per_sample_weights=weights.double() if weights is not None else None)


def exact(case, seed):
    kind, optim = case["kind"], case["optim"]
    d = _inputs(case, seed)
    if kind == "pull_push":
        return _pushed64(d["tables"]["table"], d["ids"], d["grads"], optim)
    if kind == "combine":
        return [_pushed64(t, i, g, optim) for t, i, g in zip(d["tables"].values(), d["ids"], d["grads"])][::2]
    if kind == "bags":
        lens = d["offsets"][1:] - d["offsets"][:-1]
        out = _pool64(d["tables"]["bag"], d["ids"], d["offsets"], d["bag_weights"])
        if case["mode"] == "mean":
            out = out / lens.clamp(min=1).unsqueeze(1)
        out[lens == 0] = 0.25
        return out

    params = {k: v["val"].double().requires_grad_() for k, v in d["weights"]}
    prefix = "" if kind == "mlp" else "mlp."
    with torch.no_grad():
        if kind == "mlp":
            x, wide = d["dense"].double(), 0.0
        else:
            B, F, dim = case["batch"], case["fields"], case["dim"]
            if kind == "deepfm":
                if case["fold"]:
                    rows = _rows64(d["tables"]["embedding_and_first_order"], d["ids"])
                    e, w = rows[..., :dim], rows[..., dim]
                else:
                    e = _rows64(d["tables"]["second_order"], d["ids"])
                    w = _rows64(d["tables"]["first_order"], d["ids"]).squeeze(-1)
                s = e.sum(1)
                wide = w.sum(1) + 0.5 * (s * s - (e * e).sum(1)).sum(1)
            elif kind == "wide_deep":
                e = _rows64(d["tables"]["deep"], d["ids"])
                wide = _rows64(d["tables"]["wide"], d["ids"]).sum((1, 2))
            else:
                e = _pool64(d["tables"]["combined"], d["ids"], d["offsets"]).view(B, F, dim)
                lens = (d["offsets"][1:] - d["offsets"][:-1]).view(B, F, 1)
                e[:, ::2] /= lens[:, ::2]
                wide = _pool64(d["tables"]["wide"], d["ids"], d["offsets"]).view(B, F).sum(1)
            x = torch.cat([e.reshape(B, F * dim), d["dense"].double()], 1)
            x = torch.nn.functional.pad(x, (0, d["sizes"][0] - x.shape[1]))
    h, last = x, len(d["sizes"]) - 2
    for i in range(last + 1):
        h = h @ params[f"{prefix}layers.{i}.weight"].t() + params[f"{prefix}layers.{i}.bias"]
        h = torch.relu(h) if i < last else h
    logits = h
    if kind != "mlp":
        logits = h.squeeze(-1) + wide + (params["bias"] if "bias" in params else 0.0)
    if not case.get("train", True):
        return logits.detach()
    if kind == "mlp" and case["classes"] > 1:
        loss = torch.nn.functional.cross_entropy(logits, d["labels"])
    else:
        loss = torch.nn.functional.binary_cross_entropy_with_logits(logits.reshape(-1), d["labels"].double())
    grads = torch.autograd.grad(loss, list(params.values()))
    new = {}
    for (name, value), g in zip(d["weights"], grads):
        if case.get("dct") and g.numel() >= 256:  # only the quarter of largest magnitude is sent
            kept = int(g.numel() * (1.0 - 0.75))
            tau = g.abs().reshape(-1).topk(kept).values[-1]
            g = torch.where(g.abs() >= tau, g, torch.zeros_like(g))
        new[name] = _update64(optim, _LR[optim], g, value["val"].double(), value["states"], _STEPS)
    return {"loss": loss.detach(), "logits": logits.detach(), "weights": new}
