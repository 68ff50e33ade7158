"""Workloads of the structured-loss / decoding path, by what they are in use, with their inputs and work.

A case is a dict of sizes.  Its ``kind`` says which of the framework's entry points the program calls:

* ``train``      — ``runtime.LossStep``: emissions from the decoder states, PCFG loss, both gradients, statistics;
* ``train_full`` — the fused operators under autograd, as batches of ever other shapes use them: transitions from the
  link features, emissions from the decoder states, loss, and the gradients of the model's own tensors;
* ``glat``       — a glancing training step: ``runtime.GlanceStep`` under no_grad, then ``runtime.LossStep`` on the
  second decoder pass with the revealed nodes forced to emit;
* ``glance``     — ``runtime.GlanceStep`` alone;
* ``decode``     — ``runtime.DecodeStep``, Viterbi or lookahead, from the transitions;
* ``ops_decode`` — the fused operators one by one: transitions from the link features, best tokens, lookahead decoding;
* ``ops_train``  — the operators with the reference's names on materialised logits, under autograd;
* ``ops_glance`` — the same operators under no_grad: emissions and best tree.

Lengths: sources of ``src_min`` to ``src_max`` tokens spread evenly over the batch (shuffled by the seed), a graph of
``upsample`` x source + ``offset`` nodes, a target of the source's length +-20 %; the tensors are padded to the longest
as a bucketed batch is.  Decoder states are noise plus the projection row of the token that the node is aligned with, with
a weight between 4 and 12 that differs from sentence to sentence: emissions between hardly trained and confident.
"""
import functools
import importlib.util
import math
import os
import sys

import torch
import torch.nn.functional as F

PAD, UNK, EOS = 1, 3, 2
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package of the repository that the program runs in (its directory's name is not an identifier)."""
    name = "pcfg_nat_b200"
    if name not in sys.modules:
        home = os.path.join(os.getcwd(), "pcfg-nat_b200")
        home = home if os.path.isdir(home) else os.path.join(ROOT, "pcfg-nat_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(home, "__init__.py"),
                                                      submodule_search_locations=[home])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _modules():
    _package()
    return (importlib.import_module("pcfg_nat_b200.runtime"),
            importlib.import_module("pcfg_nat_b200.custom_ops.pcfg_loss"))


def _case(name, kind, batch, src_min, src_max, upsample=4, offset=0, vocab=40000, hidden=512, **more):
    return dict(name=name, kind=kind, batch=batch, src_min=src_min, src_max=src_max, upsample=upsample, offset=offset,
                vocab=vocab, hidden=hidden, **more)


def listed():
    return [
        # the smallest call: a toy model's batch of two sentences, graph 32, vocabulary 1000 (launches and latency)
        _case("train_tiny", "train", 2, 8, 8, vocab=1000, hidden=64),
        # one training batch of 2730 target tokens
        _case("train_batch", "train", 90, 20, 40),
        # the same batch with the graph that the model builds, 8 x source + 2 nodes
        _case("train_model_graph", "train", 90, 20, 40, upsample=8, offset=2),
        # few long sentences, graph 512 and up to 154 target tokens: the dynamic program's chain is the longest
        _case("train_long", "train", 8, 96, 128),
        # the whole training step on the model's graph, from the features to their gradients and the weight's
        _case("train_full", "train_full", 90, 20, 40, upsample=8, offset=2),
        # a glancing training step (both passes) on the training batch
        _case("glat_batch", "glat", 90, 20, 40),
        # the alignment of a glancing pass: 64 sentences, graph 256
        _case("glance", "glance", 64, 64, 64),
        # interactive decoding of one sentence
        _case("decode_one", "decode", 1, 35, 35, strategy="viterbi"),
        # offline decoding, mixed lengths
        _case("decode_batch", "decode", 64, 10, 60, strategy="viterbi"),
        # lookahead decoding with the transitions formed from the link features
        _case("decode_lookahead", "ops_decode", 64, 10, 60, strategy="lookahead"),
        # an unmodified criterion: half-precision logits through the drop-in operators, forward and backward
        _case("ops_train", "ops_train", 90, 20, 40, dtype="float16"),
        # the same criterion's glancing pass in single precision, half the batch
        _case("ops_glance", "ops_glance", 45, 20, 40, dtype="float32"),
    ]


def draw(rng):
    log_int = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["train", "train", "train", "train_full", "glat", "glance", "decode", "decode",
                       "ops_decode", "ops_train", "ops_glance"])
    upsample, offset = rng.choice([(4, 0), (4, 2), (8, 2)]) if kind in ("train", "train_full", "decode", "ops_decode") else (4, 0)
    src_max = log_int(6, 128 if upsample == 4 and kind in ("train", "decode") else 64)
    src_min = max(5, int(src_max * rng.uniform(0.2, 1.0)))
    # a batch holds at most 2730 target tokens, as one of the listed ones
    most = max(1, min(128, 2730 // max(1, (src_min + src_max) // 2), 90 * 40 // src_max))
    batch = log_int(1, most)
    vocab = log_int(1000, 40000)
    if rng.random() < 0.7:
        vocab = vocab // 8 * 8  # dictionaries are usually padded to a multiple of 8
    case = dict(kind=kind, batch=batch, src_min=min(src_min, src_max), src_max=src_max, upsample=upsample, offset=offset,
                vocab=vocab, hidden=rng.choice([64, 128, 256, 512, 512]))
    if kind == "decode":
        case["strategy"] = rng.choice(["viterbi", "viterbi", "lookahead"])
    if kind == "ops_decode":
        case["strategy"] = rng.choice(["lookahead", "greedy"])
    if kind in ("ops_train", "ops_glance"):
        case["dtype"] = rng.choice(["float16", "float32"])
        if case["dtype"] == "float32":  # bounded by the listed half-precision one
            case["batch"] = max(1, batch // 2)
    return case


def _sources(case):
    B, lo, hi = case["batch"], case["src_min"], case["src_max"]
    return [hi - (hi - lo) * i // max(1, B - 1) for i in range(B)]


def _sizes(case):
    """Padded sizes (B, L, T): the longest sentence of the batch."""
    L = case["upsample"] * case["src_max"] + case["offset"]
    return case["batch"], L, max(2, min(int(1.2 * case["src_max"]), L - 2))


def _heads(case):
    return max(1, case["hidden"] // 64), 64


@functools.lru_cache(maxsize=64)
def _masks(L, device):
    """The support tree's masks as a model keeps them: left and right children [L, L], 1 = not allowed; main chain [L]."""
    return tuple(m.to(device).ne(0).to(torch.uint8) for m in _package().support_tree.get_mask(L, 1))


def _links(g, out_len, L):
    """N(0, 1) transition logits masked by the support tree, jointly log-softmaxed over (left option, right child)."""
    dev = out_len.device
    left, right, main = (m.bool() for m in _masks(L, dev))
    pos = torch.arange(L, device=dev)
    pad = pos[None, :] >= out_len[:, None]
    right_bad = pad[:, None, :] | right[None] | ~main[None, None, :]
    option = torch.stack([torch.zeros_like(pos), (pos - 1).clamp(min=0)], 1)  # node of left option k: none (0), a - 1
    left_bad = left[pos[:, None], option][None] | pad[:, option]
    bad = left_bad[:, :, :, None] | right_bad[:, :, None, :]
    x = torch.randn(bad.shape, generator=g, device=dev).masked_fill_(bad, float("-inf")).flatten(2)
    none = torch.isinf(x).all(-1, keepdim=True)
    x = torch.log_softmax(x.masked_fill(none, 0.0), -1).masked_fill(none | pad[:, :, None], float("-inf"))
    return x.view(bad.shape).contiguous()


def prepare(case, seed):
    runtime, _ = _modules()
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(dev).manual_seed(seed)
    rand = lambda *shape: torch.randn(*shape, generator=g, device=dev)  # noqa: E731
    kind, (B, L, T), V, H = case["kind"], _sizes(case), case["vocab"], case["hidden"]
    src = torch.tensor(_sources(case), device=dev)[torch.randperm(B, generator=g, device=dev)]
    out_len = src * case["upsample"] + case["offset"]
    tgt_len = torch.round(src * (0.8 + 0.4 * torch.rand(B, generator=g, device=dev))).long()
    tgt_len = torch.minimum(tgt_len.clamp(min=2, max=T), out_len - 2)
    at_t, at_l = torch.arange(T, device=dev)[None, :], torch.arange(L, device=dev)[None, :]
    targets = torch.randint(4, V, (B, T), generator=g, device=dev)
    targets = targets.masked_fill(at_t == tgt_len[:, None] - 1, EOS).masked_fill(at_t >= tgt_len[:, None], PAD)
    weight = (rand(V, H) * 0.02).half()
    aligned = targets.gather(1, (at_l * tgt_len[:, None] // out_len[:, None]).clamp(max=T - 1))
    confidence = 4.0 + 8.0 * torch.rand(B, 1, 1, generator=g, device=dev)

    def states():
        return (rand(B, L, H) + confidence / (4e-4 * H) * weight[aligned].float()).half()

    real = at_l < out_len[:, None]
    prev = torch.where(real, UNK, PAD)
    s = {"kind": kind, "seed": seed}
    if kind in ("train_full", "ops_decode"):
        heads, dim = _heads(case)
        s.update(features=[rand(B, L, heads, dim).half() for _ in range(3)] + [rand(B, L, heads)], prev=prev,
                 masks=_masks(L, dev), hidden=states(), weight=weight, output_length=out_len, targets=targets,
                 target_length=tgt_len, strategy=case.get("strategy"))
        s["n_rows"] = sum(case["upsample"] * x + case["offset"] for x in _sources(case))  # a data loader knows it
        if kind == "train_full":
            for t in (s["hidden"], s["weight"], *s["features"]):
                t.requires_grad_()
    elif kind == "train":
        s["step"] = runtime.LossStep(weight, B, L, T, dev)
        s["inputs"] = [states(), _links(g, out_len, L), out_len, targets, tgt_len]
        s["step"].run()  # the step is set up and captured before the first batch comes
    elif kind in ("glance", "glat"):
        links = _links(g, out_len, L)
        s["glance"] = runtime.GlanceStep(weight, B, L, T, dev)
        s["inputs"] = [states(), links, out_len, targets, tgt_len, prev]
        s["glance"].run()
        if kind == "glat":
            s["step"] = runtime.LossStep(weight, B, L, T, dev, force_emit=True)
            s["second"] = states()  # the decoder's second pass, over the glanced input
            s["step"].run()
    elif kind == "decode":
        s["step"] = runtime.DecodeStep(weight, B, L, _masks(L, dev)[0], dev, strategy=case["strategy"])
        s["inputs"] = [states(), _links(g, out_len, L), out_len]
        s["step"].run()
    else:
        dtype = getattr(torch, case["dtype"])
        h, w = states().to(dtype), weight.to(dtype)
        s.update(links=_links(g, out_len, L), output_length=out_len, targets=targets, target_length=tgt_len)
        if kind == "ops_train":
            s.update(hidden=h.requires_grad_(), weight=w.requires_grad_())
            s["links"].requires_grad_()
        else:
            s["logits"] = F.linear(h, w)  # the model's output of the first pass
    return s


def _emissions(s, logits, ops):
    """log P(target | node) with the criterion's end-of-sentence mask (its own element-wise operators)."""
    B, L, T = logits.shape[0], logits.shape[1], s["targets"].shape[1]
    _, match = ops.dag_logsoftmax_gather_inplace(logits, s["targets"][:, None, :].expand(-1, L, -1))
    last_t = torch.arange(T, device=match.device)[None, None, :] == (s["target_length"] - 1)[:, None, None]
    last_l = torch.arange(L, device=match.device)[None, :, None] == (s["output_length"] - 1)[:, None, None]
    return match.masked_fill(last_t & ~last_l, float("-inf"))


def run(s):
    _, ops = _modules()
    kind = s["kind"]
    if kind in ("train", "decode"):
        s["step"].load(*s["inputs"])
        return s["step"].run()
    if kind in ("glance", "glat"):
        torch.cuda.manual_seed(s["seed"])  # a trainer seeds every update, so that it can be repeated
        s["glance"].load(*s["inputs"])
        out = s["glance"].run()
        if kind == "glat":
            _, links, out_len, targets, tgt_len, _ = s["inputs"]
            s["step"].load(s["second"], links, out_len, targets, tgt_len, out[3]["matchmask"], out[3]["keep_word_mask"])
            out = (out, s["step"].run())
        return out
    if kind == "ops_train":
        match = _emissions(s, F.linear(s["hidden"], s["weight"]), ops)
        loss = ops.cuda_pcfg_loss(match, s["links"], s["output_length"], s["target_length"])
        total = -(loss / s["target_length"]).sum() * 128.0  # the trainer's loss scale
        return (loss.detach(), *torch.autograd.grad(total, (s["hidden"], s["weight"], s["links"])))
    if kind == "train_full":
        kernel = ops.get_pcfg_kernel()
        links = kernel.extract_links(*s["features"], s["prev"], PAD, *s["masks"])
        match = ops.proj_logsoftmax_gather_with_grad(s["hidden"], s["weight"], s["targets"], s["output_length"],
                                                     s["target_length"], n_rows=s["n_rows"])
        loss = ops.cuda_pcfg_loss(match, links, s["output_length"], s["target_length"])
        total = -(loss / s["target_length"]).sum() * 128.0
        return (loss.detach(), *torch.autograd.grad(total, (s["hidden"], s["weight"], *s["features"])))
    if kind == "ops_decode":
        kernel = ops.get_pcfg_kernel()
        with torch.no_grad():
            links = kernel.extract_links(*s["features"], s["prev"], PAD, *s["masks"])
            best = ops.proj_logsoftmax_gather(s["hidden"], s["weight"], None, s["output_length"], None, want_max=True)
            return kernel.lookahead_decode_device(links, best["max_lprob"], best["argmax"], s["output_length"],
                                                  s["masks"][0], PAD, 1.0, s["strategy"])
    with torch.no_grad():
        match = _emissions(s, s["logits"], ops)
        return (match, *ops.cuda_pcfg_best_tree(match, s["links"], s["output_length"], s["target_length"]))


def work(case):
    kind, (B, L, T), V, H = case["kind"], _sizes(case), case["vocab"], case["hidden"]
    sources = _sources(case)
    nodes = [case["upsample"] * x + case["offset"] for x in sources]
    rows = sum(nodes)
    proj = 2.0 * rows * H * V
    proj_bytes = 2.0 * rows * H + 2.0 * V * H
    finite_links = 4.0 * sum(2 * (m // 2) ** 2 // 2 for m in nodes)  # two left options, right children after the node
    dp = sum(4.0 * x * (m // 2) ** 2 / 2 for m, x in zip(nodes, sources))  # two products per (node, child, position)
    dense_grads = 4.0 * B * L * T + 4.0 * B * L * 2 * L
    feature_bytes, scores = 0.0, 0.0
    if kind in ("train_full", "ops_decode"):
        heads, dim = _heads(case)
        feature_bytes = 3.0 * 2 * rows * heads * dim  # query, two keys
        scores = sum(2.0 * 2 * (m // 2) ** 2 / 2 * heads * dim for m in nodes)  # two products over the triangle
    if kind == "train":
        return {"bytes": proj_bytes + finite_links + dense_grads, "flops": proj + 3 * dp}
    if kind == "train_full":  # gradients of features, states and weight, all in half precision
        grads = 3.0 * 2 * B * L * heads * dim + 2.0 * B * L * H + 2.0 * V * H
        return {"bytes": proj_bytes + feature_bytes + grads, "flops": 3 * proj + 3 * dp + 3 * scores}
    if kind == "glance":
        return {"bytes": proj_bytes + finite_links + 8.0 * B * L * 4 + B * L * T, "flops": proj + dp}
    if kind == "glat":
        return {"bytes": 2 * proj_bytes + 2 * finite_links + 8.0 * B * L * 4 + 2.0 * B * L * T + dense_grads,
                "flops": 2 * proj + 4 * dp}
    if kind == "decode":  # Viterbi: a quarter of the nodes as lengths, one max-plus term each for (node, child)
        lengths = sum(2.0 * (m // 4) * (m // 2) ** 2 / 2 for m in nodes) if case["strategy"] == "viterbi" else 0.0
        return {"bytes": proj_bytes + finite_links + 8.0 * B * L, "flops": proj + lengths}
    if kind == "ops_decode":
        return {"bytes": proj_bytes + feature_bytes + 8.0 * B * L, "flops": proj + scores}
    size = 2.0 if case["dtype"] == "float16" else 4.0
    if kind == "ops_train":  # logits written, read and overwritten by the softmax, then by their gradient, and read twice
        return {"bytes": size * (5.0 * B * L * V + 2.0 * (B * L + V) * H) + finite_links + 8.0 * B * L * L,
                "flops": 3 * 2.0 * B * L * H * V + 3 * dp}
    return {"bytes": size * B * L * V + finite_links + 4.0 * B * L * T + 8.0 * B * L, "flops": dp}


def tolerance(case):
    """About four times what was measured: the fused steps against projections in float64 and the log-space kernels,
    the autograd chains against float64 products.  In the discrete outputs nothing differed; the shares are for ties."""
    kind = case["kind"]
    if kind in ("decode", "ops_decode"):
        return {"rel": 1e-5, "differ": 5e-3}
    if kind in ("glance", "ops_glance"):
        return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
    if kind == "train_full":  # bf16 gradients of the logits, half-precision results
        return {"rel": 1e-2, "max": 0.4}
    if kind == "ops_train" and case["dtype"] == "float16":
        return {"rel": 3.2e-3, "max": 0.12}
    # single precision: the rounding of log-space sums, whose magnitude grows with the target's length
    return {"rel": 6e-5 if case["src_max"] <= 48 else 5e-4, "max": 4e-4 if case["src_max"] <= 48 else 1.5e-3, "differ": 1e-3}
