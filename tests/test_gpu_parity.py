"""GPU parity tests: the CUDA kernels, called through the C ABI (ctypes -> libpcfgnat.so), against
the CPU oracle on the same seeded inputs, against the golden outputs of the reference kernels and,
when the reference build is present next to the oracle, against the reference kernels live.

Tolerances (from the parity contract): loss 1e-4 relative, gradients 1e-3 relative, Viterbi and
best-tree indices bit-exact including tie-breaks.  The inside table is additionally required to be
bit-identical to the reference kernel's table (GPU vs GPU), because best-tree compares sums of it.
"""
import os

import numpy as np
import pytest
import torch

import oracle
import _pyref as pyref
from conftest import golden_path

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(params=["auto", "cluster", "balanced", "rows"])
def dp_kernel(request, monkeypatch):
    """Runs a test once per selection of inside/outside kernels (PCFGNAT_DP_KERNEL): the library's own
    choice by shape, warp-per-node clusters, phase-balanced single CTA, and 4 lanes per node (the only
    one without a size limit)."""
    if request.param == "auto":
        monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    else:
        monkeypatch.setenv("PCFGNAT_DP_KERNEL", request.param)
    return request.param


@pytest.fixture(params=["auto", "rows", "cluster1", "cluster4"])
def vit_kernel(request, monkeypatch):
    """Runs a Viterbi test once per kernel: the library's own choice of cluster size, the single-CTA kernel
    that reads links from global memory, and fixed clusters of 1 and 4 CTAs per sentence."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    if request.param == "rows":
        monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    elif request.param.startswith("cluster"):
        monkeypatch.setenv("PCFGNAT_DP_CLUSTER_SIZE", request.param[len("cluster"):])
    return request.param


def _g(name):
    p = golden_path(name)
    if not os.path.isfile(p):
        pytest.skip(f"{name} not recorded yet")
    return np.load(p)


def _cu(x, dtype=None):
    t = torch.as_tensor(np.ascontiguousarray(x)).to(DEV)
    return t if dtype is None else t.to(dtype)


def _bits(x):
    return np.ascontiguousarray(x).view(np.int32)


def _loss_inputs(syn, w, seed):
    b = syn.make_batch(w, seed=seed)
    return b, syn.reference_match_all(b)


def _rel_close(a, b, rtol, atol=0.0):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    fin = np.isfinite(a)
    err = np.abs(a[fin] - b[fin])
    assert (err <= atol + rtol * np.abs(b[fin])).all(), float(err.max())


CASES = [
    ("tiny", dict(batch=2, vocab=100, hidden=8, fixed_graph=32, fixed_target=10), 0),
    ("ragged", dict(batch=7, vocab=100, hidden=8, src_min=2, src_max=21), 1),
    ("mid", dict(batch=4, vocab=100, hidden=8, src_min=30, src_max=40), 2),
    ("wide", dict(batch=2, vocab=100, hidden=8, fixed_graph=256, fixed_target=40), 3),
    ("global_links", dict(batch=2, vocab=100, hidden=8, fixed_graph=400, fixed_target=30), 4),
]


@pytest.mark.parametrize("name,kw,seed", CASES)
def test_loss_forward_against_oracle(dp_kernel, monkeypatch, ops, syn, name, kw, seed):
    b, ma = _loss_inputs(syn, syn.Workload(name, emissions="logits", **kw), seed)
    k = ops.get_pcfg_kernel()
    S, C = k.pcfg_loss(ma.to(DEV), b.links.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV), 1)
    So, Co = oracle.pcfg_loss(ma.numpy(), b.links.numpy(), b.output_length.numpy(), b.target_length.numpy())
    _rel_close(S.cpu().numpy(), So, 1e-5, 1e-5)
    assert np.array_equal(_bits(C.cpu().numpy()), _bits(Co))
    _rel_close(S[:, 0, 0].cpu().numpy(), So[:, 0, 0], 1e-4)
    # the fused forward + backward keeps its table to itself, so by default it builds it in free summation
    # order (loss equal to a few ulp); with a kernel family forced, or PCFGNAT_EXACT_ORDER=1, bit for bit
    loss = ops.cuda_pcfg_loss(ma.to(DEV), b.links.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV))
    if dp_kernel == "auto":
        _rel_close(loss.cpu().numpy(), S[:, 0, 0].cpu().numpy(), 1e-5)
        monkeypatch.setenv("PCFGNAT_EXACT_ORDER", "1")
        loss = ops.cuda_pcfg_loss(ma.to(DEV), b.links.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV))
    assert np.array_equal(_bits(loss.cpu().numpy()), _bits(S[:, 0, 0].cpu().numpy()))


@pytest.mark.parametrize("name,kw,seed", CASES)
def test_loss_backward_against_oracle(dp_kernel, ops, syn, name, kw, seed):
    b, ma = _loss_inputs(syn, syn.Workload(name, emissions="logits", **kw), seed)
    ol, tl = b.output_length.numpy(), b.target_length.numpy()
    So, Co = oracle.pcfg_loss(ma.numpy(), b.links.numpy(), ol, tl)
    go = np.linspace(0.5, 2.0, b.B).astype(np.float32)
    mgo, lgo = oracle.pcfg_loss_backward(go, So, Co, ma.numpy(), b.links.numpy(), ol, tl)
    k = ops.get_pcfg_kernel()
    S, C = k.pcfg_loss(ma.to(DEV), b.links.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV), 1)
    mg, lg = k.pcfg_loss_backward(_cu(go), S, C, ma.to(DEV), b.links.to(DEV), b.output_length.to(DEV),
                                  b.target_length.to(DEV), 1)
    np.testing.assert_allclose(mg.cpu().numpy(), mgo, rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy(), lgo, rtol=1e-3, atol=2e-6)
    # fused entry point and the autograd wrapper give the same gradients (scaled by grad_output)
    mat = ma.to(DEV).requires_grad_(True)
    lkt = b.links.to(DEV).requires_grad_(True)
    loss = ops.cuda_pcfg_loss(mat, lkt, b.output_length.to(DEV), b.target_length.to(DEV))
    fin = torch.isfinite(loss)
    (loss[fin] * _cu(go)[fin]).sum().backward()
    fin_np = fin.cpu().numpy()
    np.testing.assert_allclose(mat.grad.cpu().numpy()[fin_np], mgo[fin_np], rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lkt.grad.cpu().numpy()[fin_np], lgo[fin_np], rtol=1e-3, atol=2e-6)


@pytest.fixture(params=["staged", "global"])
def tree_walk(request, monkeypatch):
    """Both best-tree kernels: the walk over a copy of its inputs in shared memory (default where it fits) and the
    walk over global memory (PCFGNAT_TREE_STAGED=0, and shapes too large for shared memory)."""
    if request.param == "global":
        monkeypatch.setenv("PCFGNAT_TREE_STAGED", "0")
    else:
        monkeypatch.delenv("PCFGNAT_TREE_STAGED", raising=False)
    return request.param


@pytest.mark.parametrize("name,kw,seed", CASES)
def test_best_tree_bit_exact_on_shared_tables(ops, syn, tree_walk, name, kw, seed):
    b, ma = _loss_inputs(syn, syn.Workload(name, emissions="logits", **kw), seed)
    ol, tl = b.output_length.numpy(), b.target_length.numpy()
    So, Co = oracle.pcfg_loss(ma.numpy(), b.links.numpy(), ol, tl)
    want = oracle.pcfg_best_tree(So, Co, ma.numpy(), b.links.numpy(), ol, tl)
    got = ops.get_pcfg_kernel().pcfg_best_tree(_cu(So), _cu(Co), ma.to(DEV), b.links.to(DEV), b.output_length.to(DEV),
                                               b.target_length.to(DEV), 1)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


def test_best_tree_tie_breaking(ops, tree_walk):
    # all transitions and emissions equal: every arg-max is a tie, so the result is decided by the
    # reference's lane order (0, 2, 1, 3), then smallest right child, then "no left child" first
    B, L, T = 1, 40, 9
    ma = np.zeros((B, L, T), np.float32)
    ma[0, :, T - 1] = -np.inf
    ma[0, L - 1, T - 1] = 0.0
    lk = np.full((B, L, 2, L), -np.inf, np.float32)
    for a in range(1, L - 1, 2):
        lk[0, a, 0, a + 2::2] = -1.0
        if a >= 3:
            lk[0, a, 1, a + 2::2] = -1.0
    ol, tl = np.array([L]), np.array([T])
    So, Co = oracle.pcfg_loss(ma, lk, ol, tl)
    So = np.where(np.isfinite(So), np.float32(-3.0), So)  # flatten the table: exact ties everywhere
    want = oracle.pcfg_best_tree(So, Co, ma, lk, ol, tl)
    got = ops.get_pcfg_kernel().pcfg_best_tree(_cu(So), None, _cu(ma), _cu(lk), _cu(ol), _cu(tl), 1)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert (want >= 0).sum() >= 2


@pytest.mark.parametrize("name", ["ref_loss_tiny.npz", "ref_loss_ragged.npz", "ref_loss_mid.npz"])
def test_loss_against_reference_golden(dp_kernel, ops, name):
    g = _g(name)
    k = ops.get_pcfg_kernel()
    ma, lk, ol, tl = _cu(g["match_all"]), _cu(g["links"]), _cu(g["output_length"]), _cu(g["target_length"])
    S, C = k.pcfg_loss(ma, lk, ol, tl, 1)
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(g["S"]))  # bit-identical to the reference kernel
    assert np.array_equal(_bits(C.cpu().numpy()), _bits(g["C"]))
    mg, lg = k.pcfg_loss_backward(torch.ones(len(ol), device=DEV), S, C, ma, lk, ol, tl, 1)
    np.testing.assert_allclose(mg.cpu().numpy(), g["match_all_grad"], rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy(), g["links_grad"], rtol=1e-3, atol=2e-6)
    tree, loss = ops.cuda_pcfg_best_tree(ma, lk, ol, tl)
    np.testing.assert_array_equal(tree.cpu().numpy(), g["tree"])
    assert np.array_equal(_bits(loss.cpu().numpy()), _bits(g["S"][:, 0, 0]))


VCASES = [
    ("v_ragged", dict(batch=6, vocab=80, hidden=8, src_min=2, src_max=20), 0),
    ("v_mid", dict(batch=3, vocab=80, hidden=8, src_min=40, src_max=60), 1),
    ("v_global_links", dict(batch=2, vocab=80, hidden=8, fixed_graph=400), 2),
    ("v_many", dict(batch=93, vocab=40, hidden=8, src_min=2, src_max=30), 3),  # mixed cluster widths by default
]


def _viterbi_inputs(syn, name, kw, seed):
    b = syn.make_batch(syn.Workload(name, emissions="logits", kind="viterbi", **kw), seed=seed)
    ob, tok = torch.log_softmax(b.logits, -1).max(-1)
    return b, ob.contiguous(), tok.contiguous()


@pytest.mark.parametrize("name,kw,seed", VCASES)
def test_viterbi_bit_exact_against_oracle(vit_kernel, ops, syn, name, kw, seed):
    b, ob, tok = _viterbi_inputs(syn, name, kw, seed)
    S, R, Lt, Mt = ops.get_pcfg_kernel().pcfg_viterbi(ob.to(DEV), b.links.to(DEV), b.output_length.to(DEV), 1)
    So, Ro, Lo, Mo = oracle.pcfg_viterbi(ob.numpy(), b.links.numpy(), b.output_length.numpy())
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(So))
    np.testing.assert_array_equal(R.cpu().numpy(), Ro)
    np.testing.assert_array_equal(Lt.cpu().numpy(), Lo)
    np.testing.assert_array_equal(Mt.cpu().numpy(), Mo)
    scores, R2, L2, M2 = ops.cuda_pcfg_viterbi(ob.to(DEV), b.links.to(DEV), b.output_length.to(DEV))
    assert np.array_equal(_bits(scores.cpu().numpy()), _bits(So[:, 1, :]))
    # length-penalised arg-max as the model does it, then the back-trace on the device
    sc = scores / torch.arange(b.L // 4, device=DEV).unsqueeze(0)
    sc.masked_fill_(sc.isnan(), float("-inf"))
    pred = sc[:, 1:].max(-1)[1] + 1
    mask = b.left_tree_mask.long()
    want = oracle.viterbi_decoding(pred.cpu().numpy(), b.output_length.numpy(), Lo, Ro, Mo, tok.numpy(), mask.numpy(), 1)
    got = ops.viterbi_decoding(pred, b.output_length.to(DEV), L2, R2, M2, tok.to(DEV), mask.to(DEV), 1)
    # the same in one launch: length choice fused into the back-trace
    pen = torch.arange(b.L // 4, device=DEV).float()
    f_tok, f_cnt, f_pred = ops.get_pcfg_kernel().viterbi_decode_device(S, pen, b.output_length.to(DEV), L2, R2, M2,
                                                                       tok.to(DEV), mask.to(DEV), 1)
    assert torch.equal(f_pred, pred)
    width = want.shape[1]
    np.testing.assert_array_equal(f_tok[:, :width].cpu().numpy(), want.astype(np.int64))
    assert (f_tok[:, width:] == 1).all() and int(f_cnt.max()) == width
    assert got.dtype == torch.float32 and got.is_cuda
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    # the reference call pattern: traces moved to the host first
    got_cpu = ops.viterbi_decoding(pred.cpu(), b.output_length, L2.cpu(), R2.cpu(), M2.cpu(), tok, mask, 1)
    assert not got_cpu.is_cuda
    np.testing.assert_array_equal(got_cpu.numpy(), want)


def test_viterbi_tie_breaking(vit_kernel, ops, syn):
    # emissions and transitions from a handful of exactly representable values: many candidates of a
    # node tie, so the backpointers are decided by the reference's scan and merge order alone
    b = syn.make_batch(syn.Workload("v_ties", emissions="logits", kind="viterbi", batch=4, vocab=80, hidden=8,
                                    src_min=10, src_max=45), seed=5)
    g = torch.Generator().manual_seed(7)
    ob = -torch.randint(1, 4, (b.B, b.L), generator=g).float() * 0.5
    finite = torch.isfinite(b.links)
    links = torch.where(finite, -torch.randint(1, 3, b.links.shape, generator=g).float() * 0.25, b.links)
    S, R, Lt, Mt = ops.get_pcfg_kernel().pcfg_viterbi(ob.to(DEV), links.to(DEV), b.output_length.to(DEV), 1)
    So, Ro, Lo, Mo = oracle.pcfg_viterbi(ob.numpy(), links.numpy(), b.output_length.numpy())
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(So))
    np.testing.assert_array_equal(R.cpu().numpy(), Ro)
    np.testing.assert_array_equal(Lt.cpu().numpy(), Lo)
    np.testing.assert_array_equal(Mt.cpu().numpy(), Mo)
    assert (np.isfinite(So).sum() > 100)


@pytest.mark.parametrize("B, L", [(1, 8), (1, 140), (3, 66), (60, 130), (100, 66), (100, 256), (150, 34), (40, 262), (5, 515),
                                  (40, 379), (38, 384), (20, 531), (5, 768), (1, 1060)])
def test_viterbi_table_and_trace_edges(ops, syn, monkeypatch, B, L):
    """Tables bit for bit those of the kernel that reads the transitions from global memory, and the back-trace the
    host restatement's, at the numbers of lanes per node, cluster sizes and shared clusters that the library picks, with
    ties, infinite and NaN transitions, short sentences and a length out of range."""
    import importlib

    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    g = torch.Generator(DEV).manual_seed(L * 3 + B)
    ob = -torch.randint(1, 6, (B, L), device=DEV, generator=g).float() / 4
    links = -torch.randint(1, 8, (B, L, 2, L), device=DEV, generator=g).float() / 4
    at = torch.arange(L, device=DEV)
    links.masked_fill_((at[None, :] <= at[:, None])[None, :, None, :], float("-inf"))
    links[0, 1, 0, 3:5], links[B // 2, 3] = float("nan"), float("-inf")
    ol = torch.randint(2, L + 1, (B,), device=DEV, generator=g)
    ol[0], ol[-1] = 2 if B > 2 else L, L
    if B > 3:
        ol[1] = L + 1
    k = ops.get_pcfg_kernel()
    got = k.pcfg_viterbi(ob, links, ol, 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    want = k.pcfg_viterbi(ob, links, ol, 1)
    assert np.array_equal(_bits(got[0].cpu().numpy()), _bits(want[0].cpu().numpy()))
    assert all(torch.equal(x, y) for x, y in zip(got[1:], want[1:])) and torch.isfinite(got[0]).any()
    ok = ol <= L
    S, R, Lt, Mt = (t[ok] for t in got)
    lm = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)[0].long()
    tok = torch.randint(1, 9, (int(ok.sum()), L), device=DEV, generator=g)
    pen = torch.arange(L // 4, device=DEV).float()
    ops.read_status(DEV)
    out, cnt, pred = k.viterbi_decode_device(S, pen, ol[ok], Lt, R, Mt, tok, lm.to(DEV), 1)
    host = [t.cpu().numpy() for t in (pred, ol[ok], Lt, R, Mt, tok)]
    for i in range(len(pred)):
        row = oracle.viterbi_decoding(*[t[i:i + 1] for t in host], lm.numpy(), 1)[0].astype(np.int64)
        assert int(cnt[i]) == len(row) and out[i].cpu().tolist() == row.tolist() + [1] * (L - len(row))
    assert ops.read_status(DEV) == 0


@pytest.mark.parametrize("B, L", [(2, 36), (9, 514), (9, 600), (40, 98), (70, 150), (260, 70), (600, 34)])
def test_viterbi_signed_zeros_and_crowded_grids(ops, monkeypatch, B, L):
    """Values that compare equal but differ in their bits (-0 and +0, of which the first in the reference's order is kept), few
    distinct values, chains beyond the terms held in registers and grids larger than the GPU: tables bit for bit those of the
    kernel that reads the transitions from global memory."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    g = torch.Generator(DEV).manual_seed(L + B)
    signed = lambda *shape: torch.randint(0, 2, shape, device=DEV, generator=g).float() * -0.0  # noqa: E731
    ob, links = signed(B, L), signed(B, L, 2, L)
    ob = torch.where(torch.rand(B, L, device=DEV, generator=g) < 0.3, -0.25, ob)
    links = torch.where(torch.rand(B, L, 2, L, device=DEV, generator=g) < 0.5, -0.5, links)
    at = torch.arange(L, device=DEV)
    links.masked_fill_((at[None, :] <= at[:, None])[None, :, None, :], float("-inf"))
    ol = torch.randint(max(2, L // 2), L + 1, (B,), device=DEV, generator=g)
    ol[0] = L
    k = ops.get_pcfg_kernel()
    got = k.pcfg_viterbi(ob, links, ol, 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    want = k.pcfg_viterbi(ob, links, ol, 1)
    assert np.array_equal(_bits(got[0].cpu().numpy()), _bits(want[0].cpu().numpy()))
    assert all(torch.equal(x, y) for x, y in zip(got[1:], want[1:])) and bool((got[0] == 0).any())
    assert ops.read_status(DEV) == 0


@pytest.mark.parametrize("B, L", [(3, 512), (2, 516), (16, 514), (24, 562), (20, 700), (1, 1060)])
def test_viterbi_of_long_chains(ops, monkeypatch, B, L):
    """Chains at and beyond 256 main-chain nodes, whose children past the first 128 are kept as a block's maximum, on the numbers
    of CTAs and lanes that the library picks for few and many sentences; few distinct values: many ties within a block and between
    blocks.  Tables bit for bit those of the kernel that reads the transitions from global memory."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    g = torch.Generator(DEV).manual_seed(L + B)
    ob = -0.25 * torch.randint(0, 3, (B, L), device=DEV, generator=g).float()
    links = -0.5 * torch.randint(0, 4, (B, L, 2, L), device=DEV, generator=g).float()
    at = torch.arange(L, device=DEV)
    links.masked_fill_((at[None, :] <= at[:, None])[None, :, None, :], float("-inf"))
    ol = torch.randint(L // 3, L + 1, (B,), device=DEV, generator=g)
    ol[0] = L
    k = ops.get_pcfg_kernel()
    got = k.pcfg_viterbi(ob, links, ol, 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    want = k.pcfg_viterbi(ob, links, ol, 1)
    assert np.array_equal(_bits(got[0].cpu().numpy()), _bits(want[0].cpu().numpy()))
    assert all(torch.equal(x, y) for x, y in zip(got[1:], want[1:]))
    assert ops.read_status(DEV) == 0


@pytest.mark.parametrize("name", ["ref_viterbi_ragged.npz", "ref_viterbi_mid.npz"])
def test_viterbi_against_reference_golden(vit_kernel, ops, name):
    g = _g(name)
    S, R, Lt, Mt = ops.get_pcfg_kernel().pcfg_viterbi(_cu(g["ob_lprob"]), _cu(g["links"]), _cu(g["output_length"]), 1)
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(g["S"]))
    np.testing.assert_array_equal(R.cpu().numpy(), g["R"])
    np.testing.assert_array_equal(Lt.cpu().numpy(), g["L"])
    np.testing.assert_array_equal(Mt.cpu().numpy(), g["M"])


def test_backtrace_against_reference_host_golden(ops):
    g = np.load(golden_path("host_viterbi_decoding.npz"))
    got = ops.viterbi_decoding(_cu(g["pred_length"]), _cu(g["output_length"]), _cu(g["L"]), _cu(g["R"]), _cu(g["M"]),
                               _cu(g["tokens"]), _cu(g["left_tree_mask"].astype(np.int64)), 1)
    np.testing.assert_array_equal(got.cpu().numpy().astype(np.int64), g["decoded"])


@pytest.fixture(params=["single", "pair"])
def proj_pair(request, monkeypatch):
    """Runs a projection test with one CTA per tile and with CTA pairs sharing every W tile (cta_group::2)."""
    monkeypatch.setenv("PCFGNAT_PROJ_PAIR", "1" if request.param == "pair" else "0")
    return request.param


@pytest.mark.parametrize("dtype,atol", [(torch.float32, 2e-5), (torch.float16, 2e-5)])
@pytest.mark.parametrize("V", [1000, 40000, 997])
def test_logsoftmax_gather_against_oracle(ops, dtype, atol, V):
    g = torch.Generator().manual_seed(V)
    B, L, slen = 2, 6, 11
    x = (torch.randn(B, L, V, generator=g) * 3).to(dtype)
    tgt = torch.randint(0, V, (B, slen), generator=g)
    sel_idx = tgt[:, None, :].expand(-1, L, -1)  # stride-0 expand, as the criterion passes it
    want, probs = oracle.logsoftmax_gather(x.float().numpy(), sel_idx.numpy(), True)
    k = ops.get_pcfg_kernel()
    xc = x.to(DEV).clone()
    got = k.logsoftmax_gather(xc, sel_idx.to(DEV), False)
    np.testing.assert_allclose(got.cpu().numpy(), want, atol=atol + 1e-4)
    assert torch.equal(xc.cpu(), x)  # untouched without require_gradient
    got2 = k.logsoftmax_gather(xc, sel_idx.to(DEV), True)
    np.testing.assert_allclose(got2.cpu().numpy(), want, atol=atol + 1e-4)
    np.testing.assert_allclose(xc.float().cpu().numpy(), probs, atol=1e-6 if dtype == torch.float32 else 1e-3,
                               rtol=1e-4 if dtype == torch.float32 else 2e-3)


@pytest.mark.parametrize("stream", ["1", "0"])
@pytest.mark.parametrize("dtype,V", [(torch.float16, 40000), (torch.float32, 8000), (torch.float32, 40000), (torch.float16, 1000)])
def test_logsoftmax_gather_several_rows_per_cta(ops, monkeypatch, stream, dtype, V):
    """More rows than CTAs: the streaming kernel refills a row's chunks with the next row's bytes while it still works
    on the row (both phases of every chunk barrier come into use); rows of one full chunk and a part, of several
    chunks, and of less than a chunk; PCFGNAT_LSG_STREAM=0 runs the single-buffer kernel instead."""
    monkeypatch.setenv("PCFGNAT_LSG_STREAM", stream)
    g = torch.Generator().manual_seed(V + 1)
    B, L, slen = 3, 250, 7
    x = (torch.randn(B, L, V, generator=g) * 3).to(dtype)
    tgt = torch.randint(0, V, (B, slen), generator=g)
    sel_idx = tgt[:, None, :].expand(-1, L, -1)
    want, probs = oracle.logsoftmax_gather(x.float().numpy(), sel_idx.numpy(), True)
    k = ops.get_pcfg_kernel()
    xc = x.to(DEV).clone()
    got = k.logsoftmax_gather(xc, sel_idx.to(DEV), False)
    np.testing.assert_allclose(got.cpu().numpy(), want, atol=1.2e-4)
    assert torch.equal(xc.cpu(), x)
    got2 = k.logsoftmax_gather(xc, sel_idx.to(DEV), True)
    np.testing.assert_allclose(got2.cpu().numpy(), want, atol=1.2e-4)
    np.testing.assert_allclose(xc.float().cpu().numpy(), probs, atol=1e-6 if dtype == torch.float32 else 1e-3,
                               rtol=1e-4 if dtype == torch.float32 else 2e-3)
    assert ops.read_status(DEV) == 0


def test_logsoftmax_gather_more_selected_columns_than_threads(ops):
    """More gathered columns per row than the streaming kernel has threads: its late gather loop, with and without
    the softmax kept; an index out of range gives NaN and the status bit in both."""
    g = torch.Generator().manual_seed(5)
    B, L, V, slen = 2, 200, 2000, 700
    x = (torch.randn(B, L, V, generator=g) * 2).half()
    tgt = torch.randint(0, V, (B, slen), generator=g)
    sel_idx = tgt[:, None, :].expand(-1, L, -1)
    want, _ = oracle.logsoftmax_gather(x.float().numpy(), sel_idx.numpy(), True)
    k = ops.get_pcfg_kernel()
    for keep in (False, True):
        got = k.logsoftmax_gather(x.to(DEV).clone(), sel_idx.to(DEV), keep)
        np.testing.assert_allclose(got.cpu().numpy(), want, atol=1.2e-4)
    assert ops.read_status(DEV) == 0
    for n_sel in (700, 9):  # the late and the early gather
        bad = tgt[:, :n_sel].clone()
        bad[1, 3] = V
        got = k.logsoftmax_gather(x.to(DEV).clone(), bad[:, None, :].expand(-1, L, -1).to(DEV), False)
        assert torch.isnan(got[1, :, 3]).all() and torch.isfinite(got[0]).all()
        assert ops.read_status(DEV) & 4  # PCFGNAT_STATUS_BAD_INDEX


def test_logsoftmax_gather_reference_golden_and_autograd(ops):
    g = _g("ref_logsoftmax_gather.npz")
    k = ops.get_pcfg_kernel()
    sel_idx = _cu(g["targets"])[:, None, :].expand(-1, 8, -1)
    for tag, dt in (("f32", torch.float32), ("f16", torch.float16)):
        x = _cu(g["logits"]).to(dt).contiguous()
        got = k.logsoftmax_gather(x, sel_idx, True)
        np.testing.assert_allclose(got.cpu().numpy(), g[f"selected_{tag}_1"], atol=1e-4)
        np.testing.assert_allclose(x.float().cpu().numpy(), g[f"probs_{tag}"], atol=1e-3 if dt == torch.float16 else 1e-6,
                                   rtol=1e-3)
    # autograd through the in-place function equals autograd through log_softmax + gather
    x0 = _cu(g["logits"])
    w = torch.randn(2, 8, 10, device=DEV, generator=torch.Generator(DEV).manual_seed(0))
    xa = x0.clone().requires_grad_(True)
    (torch.log_softmax(xa, -1).gather(2, sel_idx) * w).sum().backward()
    xb = x0.clone().requires_grad_(True)
    _, sel = ops.dag_logsoftmax_gather_inplace(xb * 1.0, sel_idx)
    (sel * w).sum().backward()
    np.testing.assert_allclose(xb.grad.cpu().numpy(), xa.grad.cpu().numpy(), atol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("V, slen", [(1, 1), (5, 3), (1003, 9), (8192, 256), (8200, 257), (40001, 40)])
def test_logsoftmax_gather_backward(ops, dtype, V, slen):
    """Rows that start off a 16-byte boundary, shorter than one block's pass and longer, repeated columns, more columns
    than threads (added atomically in the storage type), indices out of range.  One rounding of the storage type."""
    g = torch.Generator().manual_seed(V)
    B, L = 2, 5
    probs = torch.softmax(3 * torch.randn(B, L, V, generator=g), -1).to(dtype)
    idx = torch.randint(0, V, (B, L, slen), generator=g)
    idx[:, :, slen // 2:] = idx[:, :, slen // 2:] // 3  # repeated columns
    grad = torch.randn(B, L, slen, generator=g)
    want = probs.double() * -grad.double().sum(-1, keepdim=True)
    want.scatter_add_(-1, idx, grad.double())
    got = ops.get_pcfg_kernel().logsoftmax_gather_backward(probs.to(DEV), idx.to(DEV), grad.to(DEV))
    eps = 1e-3 if dtype == torch.float16 else 1e-6
    torch.testing.assert_close(got.cpu().double(), want, rtol=eps * (4 if slen > 256 else 1), atol=eps * (4 if slen > 256 else 0.01))
    ops.read_status(DEV)
    if V > 8:
        idx[1, 2, 0], idx[0, 0, slen - 1] = V, -1
        got = ops.get_pcfg_kernel().logsoftmax_gather_backward(probs.to(DEV), idx.to(DEV), grad.to(DEV))
        assert ops.read_status(DEV) & 4 and torch.isfinite(got).all()
        torch.testing.assert_close(got[1, 0].cpu().double(), want[1, 0], rtol=4 * eps, atol=4 * eps)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("V, slen", [(33, 1), (1000, 63), (2048, 64), (2049, 65), (3001, 129), (4096, 256), (4100, 255), (4104, 65)])
def test_logsoftmax_gather_backward_block_sizes(ops, dtype, V, slen):
    """Rows and column counts on both sides of the blocks' sizes, all columns repeated.  An entry is a product and sums of at
    most slen terms in float32 (half a unit, 2^-24, of the magnitudes each), rounded to the storage type once."""
    g = torch.Generator().manual_seed(V + slen)
    probs = torch.softmax(3 * torch.randn(3, 7, V, generator=g), -1).to(dtype)
    idx = torch.randint(0, max(1, slen // 3), (3, 7, slen), generator=g) * 31 % V
    grad = torch.randn(3, 7, slen, generator=g)
    exact = probs.double() * -grad.double().sum(-1, keepdim=True)
    exact.scatter_add_(-1, idx, grad.double())
    size = probs.double() * grad.double().abs().sum(-1, keepdim=True)
    size.scatter_add_(-1, idx, grad.double().abs())
    bound = (slen + 3) * 2.0 ** -24 * size + (2.0 ** -11 * exact.abs() + 2.0 ** -25 if dtype == torch.float16 else 0.0)
    got = ops.get_pcfg_kernel().logsoftmax_gather_backward(probs.to(DEV), idx.to(DEV), grad.to(DEV)).cpu()
    assert ((got.double() - exact).abs() <= bound).all()
    again = ops.get_pcfg_kernel().logsoftmax_gather_backward(probs.to(DEV), idx.to(DEV), grad.to(DEV)).cpu()
    assert torch.equal(got, again)


@pytest.mark.parametrize("slen", [256, 257, 600])
def test_logsoftmax_gather_backward_deterministic(ops, slen):
    """Under torch's deterministic algorithms the gradient repeats itself bit for bit whatever the number of columns;
    repeated columns in half precision, whose sum depends on the order."""
    g = torch.Generator().manual_seed(slen)
    B, L, V = 2, 64, 1000
    logits = (3 * torch.randn(B, L, V, generator=g)).half()
    idx = torch.randint(0, 5, (B, L, slen), generator=g).to(DEV)
    grad = (torch.randn(B, L, slen, generator=g) * torch.logspace(-3, 2, slen)).to(DEV)
    probs = torch.softmax(logits.to(DEV).double(), -1)
    want = (probs * -grad.double().sum(-1, keepdim=True)).scatter_add_(-1, idx, grad.double())

    def once():
        x = logits.to(DEV).requires_grad_()
        return torch.autograd.grad((ops.dag_logsoftmax_gather_inplace(x * 1, idx)[1] * grad).sum(), x)[0]

    torch.use_deterministic_algorithms(True)
    try:
        first = once()
        assert all(torch.equal(once(), first) for _ in range(8))
    finally:
        torch.use_deterministic_algorithms(False)
    # at most slen + 2 roundings, each of half a unit (2^-11) of at most the row's sum of magnitudes
    assert ((first.double() - want).abs() <= (slen + 2) * 2 ** -11 * grad.abs().double().sum(-1, keepdim=True)).all()


def test_fused_loss_many_sentences_mixed_cluster_widths(ops, syn, monkeypatch):
    """More sentences than half the SMs: the fused forward + backward runs its passes as cost-ordered clusters
    of two, which the costliest sentences have to themselves and the others share, one CTA each.  Loss and gradients against the oracle, with an
    invalid sentence and wildly different lengths in the batch."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    monkeypatch.delenv("PCFGNAT_EXACT_ORDER", raising=False)
    b, ma = _loss_inputs(syn, syn.Workload("many", batch=97, vocab=40, hidden=8, src_min=2, src_max=24,
                                           emissions="logits"), 21)
    ol, tl = b.output_length.clone(), b.target_length.clone()
    tl[5] = 0  # invalid: skipped, -inf loss, zero gradients
    So, Co = oracle.pcfg_loss(ma.numpy(), b.links.numpy(), ol.numpy(), tl.numpy())
    go = np.ones(b.B, np.float32)
    mgo, lgo = oracle.pcfg_loss_backward(go, So, Co, ma.numpy(), b.links.numpy(), ol.numpy(), tl.numpy())
    ops.read_status(DEV)
    loss, mg, lg = ops.get_pcfg_kernel().pcfg_loss_fwd_bwd(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV))
    want = So[:, 0, 0].copy()
    want[5] = -np.inf
    _rel_close(loss.cpu().numpy(), want, 1e-4)
    ok = np.isfinite(want)
    np.testing.assert_allclose(mg.cpu().numpy()[ok], mgo[ok], rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy()[ok], lgo[ok], rtol=1e-3, atol=2e-6)
    assert float(mg[5].abs().sum()) == 0.0 and float(lg[5].abs().sum()) == 0.0
    assert ops.read_status(DEV) & 1  # PCFGNAT_STATUS_BAD_LENGTH
    # the table-returning operator takes the same mixed widths with the reference's summation order: bit for bit
    # the table of the 4-lanes-per-node kernel (itself pinned against the reference kernels elsewhere)
    k = ops.get_pcfg_kernel()
    S_mixed, _ = k.pcfg_loss(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV), 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    S_rows, _ = k.pcfg_loss(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV), 1)
    assert np.array_equal(_bits(S_mixed.cpu().numpy()), _bits(S_rows.cpu().numpy()))
    ops.read_status(DEV)


@pytest.mark.parametrize("batch", [24, 90])
def test_fused_loss_model_graph_size(ops, syn, monkeypatch, batch):
    """Graphs of 8 * source + 2 nodes, the size the reference model builds at left_tree_layer 1
    (models/glat_decomposed_with_link_two_hands_tri_pcfg.py:322), on the sentence lengths of the training batch:
    up to 161 main-chain nodes per sentence.  Loss and gradients against the oracle, Viterbi tables bit for bit.
    With 90 sentences a chain needs two CTAs and the grid is larger than the GPU: the clusters take the sentences
    by decreasing cost; the inside table in the reference's order must not notice (bit for bit the table of the
    kernel that takes them in batch order)."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    monkeypatch.delenv("PCFGNAT_EXACT_ORDER", raising=False)
    w = syn.WORKLOADS["train_batch_model_graph"]
    b, ma = _loss_inputs(syn, syn.Workload("model_graph", batch=batch, vocab=40, hidden=8, src_min=w.src_min,
                                           src_max=w.src_max, upsample=w.upsample, graph_offset=w.graph_offset,
                                           emissions="logits"), 33)
    assert int(b.output_length.max()) > 256 and (b.output_length % 8 == 2).all()
    ol, tl = b.output_length, b.target_length
    So, Co = oracle.pcfg_loss(ma.numpy(), b.links.numpy(), ol.numpy(), tl.numpy())
    go = np.ones(b.B, np.float32)
    mgo, lgo = oracle.pcfg_loss_backward(go, So, Co, ma.numpy(), b.links.numpy(), ol.numpy(), tl.numpy())
    ops.read_status(DEV)
    k = ops.get_pcfg_kernel()
    loss, mg, lg = k.pcfg_loss_fwd_bwd(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV))
    _rel_close(loss.cpu().numpy(), So[:, 0, 0], 1e-4)
    np.testing.assert_allclose(mg.cpu().numpy(), mgo, rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy(), lgo, rtol=1e-3, atol=2e-6)
    g = torch.Generator().manual_seed(5)
    ob = torch.log_softmax(torch.randn(b.B, b.L, 50, generator=g), -1).max(-1).values.contiguous()
    So2, Ro, Lo, Mo = oracle.pcfg_viterbi(ob.numpy(), b.links.numpy(), ol.numpy())
    S2, R2, L2, M2 = k.pcfg_viterbi(ob.to(DEV), b.links.to(DEV), ol.to(DEV), 1)
    assert np.array_equal(_bits(S2.cpu().numpy()), _bits(So2))
    np.testing.assert_array_equal(R2.cpu().numpy(), Ro)
    np.testing.assert_array_equal(L2.cpu().numpy(), Lo)
    np.testing.assert_array_equal(M2.cpu().numpy(), Mo)
    S_ranked, _ = k.pcfg_loss(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV), 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    S_rows, _ = k.pcfg_loss(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV), 1)
    assert np.array_equal(_bits(S_ranked.cpu().numpy()), _bits(S_rows.cpu().numpy()))
    assert ops.read_status(DEV) == 0


@pytest.mark.parametrize("B, L, T", [(1, 2, 1), (3, 8, 5), (4, 64, 30), (20, 162, 40), (5, 515, 70), (3, 780, 200), (30, 260, 60),
                                     (60, 98, 31), (60, 255, 76), (50, 330, 100), (80, 36, 12), (100, 33, 10), (100, 129, 40),
                                     (100, 256, 76), (90, 280, 20), (150, 30, 9), (200, 66, 20), (260, 130, 30), (300, 40, 12)])
def test_inside_table_edges(ops, monkeypatch, B, L, T):
    """Tables bit for bit those of the kernel with a thread row per node, at the numbers of lanes per node, cluster sizes and
    shared clusters that the library picks, chains beyond the terms held in registers included; with NaN and infinite transitions
    and emissions, sentences without a finite term, odd, short and out-of-range lengths, one target token."""
    for name in ("PCFGNAT_DP_KERNEL", "PCFGNAT_DP_CLUSTER_SIZE"):
        monkeypatch.delenv(name, raising=False)
    g = torch.Generator(DEV).manual_seed(L * 3 + B)
    match = 2 * torch.randn(B, L, T, device=DEV, generator=g) - 6
    links = torch.randn(B, L, 2, L, device=DEV, generator=g) - 4
    at = torch.arange(L, device=DEV)
    links.masked_fill_((at[None, :] <= at[:, None])[None, :, None, :], float("-inf"))
    ol = torch.randint(max(2, L // 4), L + 1, (B,), device=DEV, generator=g)
    tl = torch.randint(1, T + 1, (B,), device=DEV, generator=g)
    ol[0], tl[0], ol[-1], tl[-1] = L, T, L, max(1, T - 1)
    if B > 3:
        links[1].masked_fill_(torch.rand(L, 2, L, device=DEV, generator=g) < 0.05, float("nan"))
        match[1].masked_fill_(torch.rand(L, T, device=DEV, generator=g) < 0.02, float("nan"))
        links[2].masked_fill_(torch.rand(L, 2, L, device=DEV, generator=g) < 0.6, float("-inf"))
        match[2, :, T // 2:] = float("-inf")
        links[3, L // 2, 0, -3:] = float("inf")
    if B > 4:
        tl[2], tl[4], ol[B // 2], tl[B // 2 + 1] = T, 1, L + 1, 0
    k = ops.get_pcfg_kernel()
    ops.read_status(DEV)
    S, C = k.pcfg_loss(match, links, ol, tl, 1)
    status = ops.read_status(DEV)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    want_S, want_C = k.pcfg_loss(match, links, ol, tl, 1)
    assert status == ops.read_status(DEV) == (B > 4)  # PCFGNAT_STATUS_BAD_LENGTH
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(want_S.cpu().numpy()))
    assert np.array_equal(_bits(C.cpu().numpy()), _bits(want_C.cpu().numpy()))
    assert torch.isfinite(S).any()


@pytest.mark.parametrize("B, L, T", [(32, 640, 12), (20, 700, 30), (24, 640, 40), (2, 1170, 40), (3, 820, 400)])
def test_inside_table_of_long_chains(ops, monkeypatch, B, L, T):
    """More CTAs than SMs, of which no two fit an SM, and the chains that the lanes of a node cannot take (a warp per node, on
    clusters of sixteen): tables bit for bit those of the kernel with a thread row per node."""
    for name in ("PCFGNAT_DP_KERNEL", "PCFGNAT_DP_CLUSTER_SIZE"):
        monkeypatch.delenv(name, raising=False)
    g = torch.Generator(DEV).manual_seed(L + B)
    match, links = 2 * torch.randn(B, L, T, device=DEV, generator=g) - 6, torch.randn(B, L, 2, L, device=DEV, generator=g) - 4
    at = torch.arange(L, device=DEV)
    links.masked_fill_((at[None, :] <= at[:, None])[None, :, None, :], float("-inf"))
    ol = torch.randint(L // 3, L + 1, (B,), device=DEV, generator=g)
    ol[0] = L
    tl = torch.randint(T // 2, T + 1, (B,), device=DEV, generator=g)
    tl[0] = T
    k = ops.get_pcfg_kernel()
    S, C = k.pcfg_loss(match, links, ol, tl, 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    want_S, want_C = k.pcfg_loss(match, links, ol, tl, 1)
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(want_S.cpu().numpy()))
    assert np.array_equal(_bits(C.cpu().numpy()), _bits(want_C.cpu().numpy()))
    assert ops.read_status(DEV) == 0 and torch.isfinite(S).any()


@pytest.mark.parametrize("batch", [97, 6])  # one CTA per sentence; a cluster of CTAs per sentence
@pytest.mark.parametrize("L_even", [True, False])
def test_outside_pass_with_fused_gradients_matches_the_gradient_kernel(ops, syn, monkeypatch, L_even, batch):
    """Fused forward + backward: the outside kernel (single-CTA or cluster family, by batch size) that also sums up
    both gradients (emission gradients from the shares the inside pass leaves in match_all_grad) against the
    outside kernel followed by the gradient kernel (PCFGNAT_FUSED_GRAD=0): both gradients to rounding, and both
    against the oracle.  The batch has odd graph lengths, a
    one-token target, an invalid sentence, and the outputs are handed over filled with garbage."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    monkeypatch.delenv("PCFGNAT_EXACT_ORDER", raising=False)
    monkeypatch.setenv("PCFGNAT_LINEAR_DP", "0")  # this test is about the log-space kernels behind the fused entry
    b, ma = _loss_inputs(syn, syn.Workload("fg", batch=batch, vocab=40, hidden=8, src_min=3, src_max=20 if batch > 6 else 60,
                                           emissions="logits"), 77)
    links = b.links
    if not L_even:  # an odd padded width: the zero fill cannot use 16-byte stores
        ma = torch.nn.functional.pad(ma, (0, 0, 0, 1), value=0.0).contiguous()
        links = torch.nn.functional.pad(links, (0, 1, 0, 0, 0, 1), value=float("-inf")).contiguous()
    ol, tl = b.output_length.clone(), b.target_length.clone()
    ol[1] -= 1  # odd number of nodes: the last token is emitted by an even node
    tl[2] = 1   # one target token
    tl[3] = 0   # invalid
    k = ops.get_pcfg_kernel()
    ops.read_status(DEV)
    outs = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("PCFGNAT_FUSED_GRAD", mode)
        # whatever the allocator hands out next is dirty
        torch.empty(64 << 20, dtype=torch.uint8, device=DEV).fill_(0x7f)
        loss, mg, lg = k.pcfg_loss_fwd_bwd(ma.to(DEV), links.to(DEV), ol.to(DEV), tl.to(DEV))
        outs[mode] = (mg.cpu().numpy(), lg.cpu().numpy(), loss.cpu().numpy())
    assert ops.read_status(DEV) & 1  # PCFGNAT_STATUS_BAD_LENGTH for sentence 3
    # the inside pass that also emits the shares adds its two kinds of terms up separately: last-bit differences
    _rel_close(outs["1"][2], outs["0"][2], 1e-6)
    np.testing.assert_allclose(outs["1"][1], outs["0"][1], rtol=1e-4, atol=1e-7)
    np.testing.assert_allclose(outs["1"][0], outs["0"][0], rtol=1e-4, atol=1e-9)  # no absolute slack
    assert not np.array_equal(outs["1"][0], outs["0"][0])  # the switch chose another kernel
    So, Co = oracle.pcfg_loss(ma.numpy(), links.numpy(), ol.numpy(), tl.numpy())
    go = np.ones(b.B, np.float32)
    mgo, lgo = oracle.pcfg_loss_backward(go, So, Co, ma.numpy(), links.numpy(), ol.numpy(), tl.numpy())
    finite = np.isfinite(So[:, 0, 0])
    finite[3] = False
    np.testing.assert_allclose(outs["1"][0][finite], mgo[finite], rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(outs["1"][1][finite], lgo[finite], rtol=1e-3, atol=2e-6)
    assert not outs["1"][0][3].any() and not outs["1"][1][3].any()
    infeasible = ~np.isfinite(outs["1"][2])
    assert not outs["1"][0][infeasible].any() and not outs["1"][1][infeasible].any()


def test_invalid_sentences_are_skipped_not_faulted(dp_kernel, ops, syn):
    b, ma = _loss_inputs(syn, syn.Workload("bad", batch=4, vocab=50, hidden=8, src_min=4, src_max=6,
                                           emissions="logits"), 9)
    ol = b.output_length.clone()
    tl = b.target_length.clone()
    ol[1] = b.L + 5  # more nodes than the graph holds
    tl[2] = 0  # empty target
    ops.read_status(DEV)
    mat, lkt = ma.to(DEV).requires_grad_(True), b.links.to(DEV).requires_grad_(True)
    loss = ops.cuda_pcfg_loss(mat, lkt, ol.to(DEV), tl.to(DEV))
    assert torch.isinf(loss[1]) and torch.isinf(loss[2]) and torch.isfinite(loss[0]) and torch.isfinite(loss[3])
    loss[[0, 3]].sum().backward()
    assert float(mat.grad[1].abs().sum()) == 0.0 and float(lkt.grad[2].abs().sum()) == 0.0
    tree, _ = ops.cuda_pcfg_best_tree(ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV))
    assert (tree[1] == -1).all() and (tree[2] == -1).all()
    assert ops.read_status(DEV) & 1  # PCFGNAT_STATUS_BAD_LENGTH
    # odd graph length: node m-1 is a leaf; the oracle restates what the reference does with it
    ol2 = b.output_length.clone()
    ol2[0] -= 1
    ol2[3] -= 1
    lp = torch.log_softmax(b.logits, -1)
    ma2 = lp.gather(2, b.targets[:, None, :].expand(-1, b.L, -1)).contiguous()
    syn.eos_mask_(ma2, ol2, b.target_length)
    S, C = ops.get_pcfg_kernel().pcfg_loss(ma2.to(DEV), b.links.to(DEV), ol2.to(DEV), b.target_length.to(DEV), 1)
    So, Co = oracle.pcfg_loss(ma2.numpy(), b.links.numpy(), ol2.numpy(), b.target_length.numpy())
    _rel_close(S.cpu().numpy(), So, 1e-5, 1e-5)
    mg, lg = ops.get_pcfg_kernel().pcfg_loss_backward(torch.ones(4, device=DEV), S, C, ma2.to(DEV), b.links.to(DEV),
                                                      ol2.to(DEV), b.target_length.to(DEV), 1)
    mgo, lgo = oracle.pcfg_loss_backward(np.ones(4, np.float32), So, Co, ma2.numpy(), b.links.numpy(), ol2.numpy(),
                                         b.target_length.numpy())
    np.testing.assert_allclose(mg.cpu().numpy(), mgo, rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy(), lgo, rtol=1e-3, atol=2e-6)
    want = oracle.pcfg_best_tree(So, Co, ma2.numpy(), b.links.numpy(), ol2.numpy(), b.target_length.numpy())
    got = ops.get_pcfg_kernel().pcfg_best_tree(_cu(So), None, ma2.to(DEV), b.links.to(DEV), ol2.to(DEV),
                                               b.target_length.to(DEV), 1)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


def test_argument_errors(ops):
    k = ops.get_pcfg_kernel()
    ma = torch.zeros(1, 10, 3, device=DEV)
    with pytest.raises(RuntimeError, match="max_left"):
        k.pcfg_loss(ma, torch.zeros(1, 10, 4, 10, device=DEV), torch.tensor([10]), torch.tensor([3]), 1)
    with pytest.raises(RuntimeError, match="float32"):
        k.pcfg_loss(ma.double(), torch.zeros(1, 10, 2, 10, device=DEV), torch.tensor([10]), torch.tensor([3]), 1)
    with pytest.raises(RuntimeError, match="config should be 1~4"):
        k.pcfg_viterbi(torch.zeros(1, 16, device=DEV), torch.zeros(1, 16, 2, 16, device=DEV), torch.tensor([16]), 7)
    with pytest.raises(RuntimeError, match="select_idx should be long"):
        k.logsoftmax_gather(torch.zeros(1, 2, 5, device=DEV), torch.zeros(1, 2, 1, device=DEV, dtype=torch.int32), False)
    with pytest.raises(RuntimeError, match="not contiguous"):
        k.logsoftmax_gather(torch.zeros(1, 5, 2, device=DEV).transpose(1, 2), torch.zeros(1, 2, 1, device=DEV, dtype=torch.long), False)


# ---- full-size workloads: properties that need no oracle run ---------------------------------------------------

@pytest.mark.parametrize("wname", ["glance", "long_seq"])
def test_full_size_properties(dp_kernel, ops, syn, wname):
    w = syn.WORKLOADS[wname]
    b = syn.make_batch(syn.Workload(w.name, batch=w.batch, vocab=64, hidden=8, fixed_graph=w.fixed_graph,
                                    fixed_target=w.fixed_target, emissions="logits"), seed=0)
    ma = syn.reference_match_all(b).to(DEV).requires_grad_(True)
    lk = b.links.to(DEV).requires_grad_(True)
    ol, tl = b.output_length.to(DEV), b.target_length.to(DEV)
    loss = ops.cuda_pcfg_loss(ma, lk, ol, tl)
    assert torch.isfinite(loss).all()
    loss.sum().backward()
    n = int(b.target_length[0])
    # posterior marginals: each target position is emitted by exactly one node
    torch.testing.assert_close(ma.grad.sum(1)[:, :n], torch.ones(b.B, n, device=DEV), rtol=0, atol=2e-3)
    # expected number of binary rule uses = expected number of main-chain nodes used - 1
    used_main = ma.grad[:, 1::2, :].sum((1, 2))
    torch.testing.assert_close(lk.grad.sum((1, 2, 3)), used_main - 1, rtol=0, atol=5e-3)
    tree, loss2 = ops.cuda_pcfg_best_tree(ma.detach(), lk.detach(), ol, tl)
    if dp_kernel == "auto":  # free-order table inside the fused forward + backward
        torch.testing.assert_close(loss2, loss.detach(), rtol=1e-5, atol=0)
    else:
        assert torch.equal(loss2, loss.detach())
    t = tree.cpu().numpy()
    for i in range(b.B):
        used = t[i][t[i] >= 0]
        assert used.tolist() == list(range(n))
        assert t[i, 1] == 0 and t[i, int(b.output_length[i]) - 1] == n - 1


def test_full_size_viterbi_properties(ops, syn):
    b = syn.make_batch(syn.Workload("v64", batch=64, vocab=64, hidden=8, src_min=10, src_max=60, emissions="logits",
                                    kind="viterbi"), seed=0)
    ob, tok = torch.log_softmax(b.logits, -1).max(-1)
    tok = torch.arange(b.L)[None, :].expand(b.B, -1).contiguous() + 100
    scores, R, Lt, Mt = ops.cuda_pcfg_viterbi(ob.to(DEV), b.links.to(DEV), b.output_length.to(DEV))
    sc = scores / torch.arange(b.L // 4, device=DEV).unsqueeze(0)
    sc.masked_fill_(sc.isnan(), float("-inf"))
    pred = sc[:, 1:].max(-1)[1] + 1
    out = ops.viterbi_decoding(pred, b.output_length.to(DEV), Lt, R, Mt, tok.to(DEV), b.left_tree_mask.long().to(DEV), 1)
    out = out.cpu().numpy()
    for i in range(b.B):
        row = out[i][out[i] != 1]
        assert len(row) == int(pred[i]) and row[0] == 101 and row[-1] == 100 + int(b.output_length[i]) - 1
        assert (np.diff(row) > 0).all()


# ---- live comparison with the reference kernels (only where the reference build travelled along) ------------------

def _ref():
    from oracle.build_ref import load_ref, ref_so_path

    if not os.path.isfile(ref_so_path()):
        pytest.skip("reference extension not built")
    return load_ref()


@pytest.mark.parametrize("seed", [10, 11, 12])
def test_live_against_reference_kernels(dp_kernel, ops, syn, seed):
    ref = _ref()
    # graph length <= 256 keeps every reference launch at one row segment per sentence (no
    # dependence on co-resident blocks in its spin-waits)
    w = syn.Workload("live", batch=8, vocab=120, hidden=8, src_min=6, src_max=64, emissions="logits")
    b, ma = _loss_inputs(syn, w, seed)
    ma_d, lk_d = ma.to(DEV), b.links.to(DEV)
    ol, tl = b.output_length.to(DEV), b.target_length.to(DEV)
    k = ops.get_pcfg_kernel()
    Sr, Cr = ref.pcfg_loss(ma_d, lk_d, ol, tl, 1)
    S, C = k.pcfg_loss(ma_d, lk_d, ol, tl, 1)
    assert torch.equal(S.view(torch.int32), Sr.view(torch.int32))
    assert torch.equal(C.view(torch.int32), Cr.view(torch.int32))
    mgr, lgr = ref.pcfg_loss_backward(torch.ones(b.B, device=DEV), Sr, Cr, ma_d, lk_d, ol, tl, 1)
    mg, lg = k.pcfg_loss_backward(torch.ones(b.B, device=DEV), S, C, ma_d, lk_d, ol, tl, 1)
    torch.testing.assert_close(mg, mgr, rtol=1e-3, atol=2e-6)
    torch.testing.assert_close(lg, lgr, rtol=1e-3, atol=2e-6)
    assert torch.equal(k.pcfg_best_tree(S, C, ma_d, lk_d, ol, tl, 1), ref.pcfg_best_tree(Sr, Cr, ma_d, lk_d, ol, tl, 1))
    ob = torch.log_softmax(b.logits, -1).max(-1)[0].to(DEV)
    for x, y in zip(k.pcfg_viterbi(ob, lk_d, ol, 1), ref.pcfg_viterbi(ob, lk_d, ol, 1)):
        assert torch.equal(x.view(torch.int32) if x.dtype == torch.float32 else x,
                           y.view(torch.int32) if y.dtype == torch.float32 else y)


# ---- fused projection + log-softmax + gather / max (tensor cores) ------------------------------------------------

def _proj_reference(hidden, weight, targets):
    """fp32 torch reference on the GPU: same fp16 values, fp32 accumulation."""
    logits = hidden.float().reshape(-1, hidden.shape[-1]) @ weight.float().t()
    lse = torch.logsumexp(logits, -1)
    lp = logits - lse[:, None]
    mx, am = lp.max(-1)
    B, L = hidden.shape[:2]
    match = lp.view(B, L, -1).gather(2, targets[:, None, :].expand(-1, L, -1)) if targets is not None else None
    top2 = logits.topk(2, -1)[0]
    return match, mx.view(B, L), am.view(B, L), lse.view(B, L), (top2[:, 0] - top2[:, 1]).view(B, L)


PROJ_CASES = [
    # B, L, T, V, H, hidden_std
    (2, 32, 10, 1000, 64, 1.0),       # tiny: one partial row tile, vocabulary split over many CTAs
    (3, 100, 17, 5000, 128, 1.0),     # rows and vocabulary both ragged against the tile sizes
    (1, 240, 12, 40000, 512, 1.0),    # batch-1 decode shape
    (6, 160, 40, 40000, 512, 0.02),   # training-shaped slice
    (4, 256, 64, 40000, 512, 1.0),    # glancing-shaped slice
]


@pytest.mark.parametrize("B,L,T,V,H,std", PROJ_CASES)
def test_fused_projection_against_torch(proj_pair, ops, syn, B, L, T, V, H, std):
    g = torch.Generator().manual_seed(B * 1000 + L)
    hidden = (torch.randn(B, L, H, generator=g) * std).half().to(DEV)
    weight = (torch.randn(V, H, generator=g) * 0.02).half().to(DEV)
    targets = torch.randint(0, V, (B, T), generator=g).to(DEV)
    targets[:, 0] = V - 1  # last vocabulary column (inside the ragged last tile)
    targets[:, 1] = targets[:, 2]  # repeated target
    ops.read_status(DEV)
    out = ops.proj_logsoftmax_gather(hidden, weight, targets, want_max=True, want_lse=True)
    match, mx, am, lse, margin = _proj_reference(hidden, weight, targets)
    # fp16 inputs, fp32 accumulation on both sides: only summation order differs
    torch.testing.assert_close(out["lse"], lse, rtol=0, atol=2e-3)
    torch.testing.assert_close(out["match"], match, rtol=0, atol=2e-3)
    torch.testing.assert_close(out["max_lprob"], mx, rtol=0, atol=2e-3)
    clear = margin > 1e-3  # arg-max must agree wherever the top-2 margin exceeds the tolerance
    assert torch.equal(out["argmax"][clear], am[clear])
    if std >= 1.0:
        assert clear.float().mean() > 0.9
    assert ops.read_status(DEV) == 0
    # gather-only and max-only variants, EOS masking fused
    ol = torch.full((B,), L, device=DEV)
    tl = torch.full((B,), T, device=DEV)
    ol[0] = L - 2
    tl[0] = max(T - 3, 2)
    out2 = ops.proj_logsoftmax_gather(hidden, weight, targets, ol, tl, want_max=True)
    want = syn.eos_mask_(match.clone(), ol.cpu(), tl.cpu())
    real = (torch.arange(L, device=DEV)[None, :] < ol[:, None])  # with lengths only real nodes are projected
    want[~real] = 0.0
    fin = torch.isfinite(want)
    assert torch.equal(fin, torch.isfinite(out2["match"]))
    torch.testing.assert_close(out2["match"][fin], want[fin], rtol=0, atol=2e-3)
    assert float(out2["match"][~real].abs().sum()) == 0.0 and float(out2["max_lprob"][~real].abs().sum()) == 0.0
    torch.testing.assert_close(out2["max_lprob"][real], mx[real], rtol=0, atol=2e-3)
    out3 = ops.proj_logsoftmax_gather(hidden, weight, want_max=True)
    assert torch.equal(out3["argmax"], out["argmax"]) and torch.equal(out3["max_lprob"], out["max_lprob"])


@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("V,H,std", [(1000, 64, 1.0), (4104, 128, 0.3), (997, 64, 1.0)])
def test_fused_projection_backward_against_torch(proj_pair, ops, syn, V, H, std, compact):
    """Gradients of the fused projection (logits recomputed on the tensor cores, bf16 d-logits, two GEMMs)
    against float32 autograd of the same expression; with the d-logits of every padded row and (compact) of the
    real graph nodes only."""
    w = syn.Workload("pb", batch=5, vocab=V, hidden=H, src_min=8, src_max=40, hidden_std=std)
    b = syn.make_batch(w, seed=V)
    g = torch.Generator().manual_seed(1)
    gm = torch.randn(b.B, b.L, b.T, generator=g)
    gm[torch.rand(b.B, b.L, b.T, generator=g) < 0.5] = 0
    hid = b.hidden.to(DEV).requires_grad_(True)
    wt = b.weight.to(DEV).requires_grad_(True)
    ol, tl = b.output_length.to(DEV), b.target_length.to(DEV)
    match = ops.proj_logsoftmax_gather_with_grad(hid, wt, b.targets.to(DEV), ol, tl,
                                                 n_rows=int(b.output_length.sum()) if compact else None)
    fin = torch.isfinite(match)
    (match[fin] * gm.to(DEV)[fin]).sum().backward()
    # float32 reference of the same expression
    h32 = b.hidden.float().to(DEV).requires_grad_(True)
    w32 = b.weight.float().to(DEV).requires_grad_(True)
    lp = torch.log_softmax(h32 @ w32.t(), -1)
    ref = lp.gather(2, b.targets.to(DEV)[:, None, :].expand(-1, b.L, -1))
    rows = torch.arange(b.L, device=DEV)[None, :] < ol[:, None]
    syn.eos_mask_(ref, ol, tl)
    ref = torch.where(rows[:, :, None], ref, torch.zeros_like(ref))  # padding nodes are not projected: zeros
    assert torch.equal(torch.isfinite(ref), fin)
    torch.testing.assert_close(match[fin], ref[fin].detach(), rtol=2e-3, atol=2e-3)
    (ref[fin] * gm.to(DEV)[fin]).sum().backward()
    for got, want in ((hid.grad.float(), h32.grad), (wt.grad.float(), w32.grad)):
        err = (got - want).norm() / want.norm()
        assert float(err) < 1.5e-2, float(err)
        assert float((got - want).abs().max()) < 3e-2 * float(want.abs().max()) + 1e-3
    assert float(hid.grad[~rows].abs().sum()) == 0.0
    assert ops.read_status(DEV) == 0


def test_loss_step_with_projection_backward_matches_autograd_path(pkg, ops, syn):
    """LossStep(proj_backward=True): d hidden and d weight (compact d-logits in the graph, the two GEMMs after it)
    against the differentiable operator fed with the step's own emission gradient; two batches with different
    numbers of real nodes through the same step object."""
    import importlib
    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("pbs", batch=6, vocab=1000, hidden=64, src_min=6, src_max=30, hidden_std=1.0)
    batches = [syn.make_batch(w, seed=seed) for seed in (31, 32)]
    B, L, T = batches[0].B, max(b.L for b in batches), max(b.T for b in batches)
    weight = batches[0].weight.to(DEV)
    step = runtime.LossStep(weight, B, L, T, DEV, use_graph=True, proj_backward=True)
    assert int(batches[0].output_length.sum()) != int(batches[1].output_length.sum())
    for b in batches:
        hidden = torch.zeros(B, L, b.hidden.shape[2], dtype=b.hidden.dtype)
        hidden[:, :b.L] = b.hidden
        links = torch.full((B, L, 2, L), float("-inf"))
        links[:, :b.L, :, :b.L] = b.links
        targets = torch.ones(B, T, dtype=torch.int64)
        targets[:, :b.T] = b.targets
        step.load(hidden, links, b.output_length, targets, b.target_length)
        stats, mg, lg, loss, d_hidden, d_weight = step.run()
        torch.cuda.synchronize()
        assert torch.isfinite(loss).all()
        hid = hidden.to(DEV).requires_grad_(True)
        wt = weight.clone().requires_grad_(True)
        ol = b.output_length.to(DEV)
        match = ops.proj_logsoftmax_gather_with_grad(hid, wt, targets.to(DEV), ol, b.target_length.to(DEV))
        fin = torch.isfinite(match)
        (match[fin] * mg[fin]).sum().backward()
        for got, want in ((d_hidden.float(), hid.grad.float()), (d_weight.float(), wt.grad.float())):
            assert float((got - want).norm() / want.norm()) < 2e-3
        rows = torch.arange(L, device=DEV)[None, :] < ol[:, None]
        assert float(d_hidden[~rows].abs().sum()) == 0.0
    assert ops.read_status(DEV) == 0


@pytest.mark.parametrize("n,V,H", [(300, 1024, 64), (1000, 4104, 512), (129, 40000, 128), (70, 200, 8)])
def test_projection_backward_gemms_against_torch(ops, n, V, H):
    """pcfgnat_proj_backward_gemms (tcgen05, dlogits read K-major for one product and MN-major for the other)
    against float32 matmul of the same bf16 operands; shapes with row, column and K tails, one tile and many."""
    g = torch.Generator().manual_seed(n)
    dl = (torch.randn(n, V, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    w = torch.randn(V, H, generator=g).to(torch.bfloat16).to(DEV)
    rows = torch.randn(n, H, generator=g).to(torch.bfloat16).to(DEV)
    k = ops.get_pcfg_kernel()
    d_rows, d_weight = k.proj_backward_gemms(dl, w, rows)
    want_rows = dl.float() @ w.float()
    want_weight = dl.float().t() @ rows.float()
    torch.testing.assert_close(d_rows, want_rows, rtol=2e-3, atol=2e-3 * float(want_rows.abs().max()))
    torch.testing.assert_close(d_weight, want_weight, rtol=2e-3, atol=2e-3 * float(want_weight.abs().max()))
    only_rows, none = k.proj_backward_gemms(dl, w, None, want_weight=False)
    assert none is None
    torch.testing.assert_close(only_rows, d_rows, rtol=1e-5, atol=1e-5 * float(want_rows.abs().max()))
    assert ops.read_status(DEV) == 0


def test_projection_backward_gemms_with_no_rows(ops):
    """A batch without real nodes: d rows is empty and d weight exactly zero."""
    k = ops.get_pcfg_kernel()
    dl = torch.empty((0, 1024), dtype=torch.bfloat16, device=DEV)
    w = torch.ones((1024, 64), dtype=torch.bfloat16, device=DEV)
    rows = torch.empty((0, 64), dtype=torch.bfloat16, device=DEV)
    d_rows, d_weight = k.proj_backward_gemms(dl, w, rows)
    assert tuple(d_rows.shape) == (0, 64) and tuple(d_weight.shape) == (1024, 64)
    assert float(d_weight.abs().sum()) == 0.0
    with pytest.raises(RuntimeError, match="unsupported"):
        k.proj_backward_gemms(torch.zeros((8, 1001), dtype=torch.bfloat16, device=DEV),
                              torch.zeros((1001, 64), dtype=torch.bfloat16, device=DEV), None, want_weight=False)


@pytest.mark.parametrize("B, L, V, H, ragged", [(1, 3, 1001, 64, False), (3, 50, 513, 128, True), (5, 70, 2047, 64, True),
                                                (2, 130, 4004, 512, False), (4, 64, 3999, 256, True), (2, 33, 33, 64, True)])
def test_projection_backward_of_a_vocabulary_that_is_no_multiple_of_eight(ops, B, L, V, H, ragged):
    """d hidden and d weight where a row of d-logits is no multiple of 16 bytes (its padding is never read), over all
    rows and over the real nodes only, against autograd in float64: bf16 d-logits and operands (2^-8 each, rounded
    independently), sums of up to 4004 terms: 1e-2 of the result's norm; single entries 3e-2 of the largest."""
    g = torch.Generator(DEV).manual_seed(V)
    hidden, weight = torch.randn(B, L, H, device=DEV, generator=g).half(), (torch.randn(V, H, device=DEV, generator=g) * 0.1).half()
    T = 6
    targets = torch.randint(0, V, (B, T), device=DEV, generator=g)
    targets[0, 0] = V - 1
    ol = torch.randint(1, L + 1, (B,), device=DEV, generator=g) if ragged else torch.full((B,), L, device=DEV)
    grad = torch.randn(B, L, T, device=DEV, generator=g)
    real = torch.arange(L, device=DEV)[None] < ol[:, None]
    h64, w64 = hidden.double().requires_grad_(), weight.double().requires_grad_()
    lp = torch.log_softmax(h64 @ w64.t(), -1).gather(2, targets[:, None].expand(-1, L, -1))
    want = torch.autograd.grad((lp * grad * real[..., None]).sum(), (h64, w64))
    for n_rows in (None, int(ol.sum())):
        h, w = hidden.clone().requires_grad_(), weight.clone().requires_grad_()
        match = ops.proj_logsoftmax_gather_with_grad(h, w, targets, ol, None, n_rows=n_rows)
        got = torch.autograd.grad(match, (h, w), grad)
        for x, y in zip(got, want):
            assert torch.isfinite(x).all() and x.shape == y.shape
            assert (x.double() - y).norm() <= 1e-2 * y.norm() and (x.double() - y).abs().max() <= 3e-2 * y.abs().max()
        assert (got[0][~real] == 0).all()


def test_loss_step_with_projection_backward_of_an_odd_vocabulary(pkg, ops, syn):
    """The step object's d hidden and d weight with padded rows of d-logits, against the differentiable operator (which the
    test above holds to float64): the same kernels over the same rows, sums by atomics in another order."""
    import importlib
    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    b = syn.make_batch(syn.Workload("odd", batch=4, vocab=1003, hidden=64, src_min=6, src_max=20, hidden_std=1.0), seed=3)
    weight = b.weight.to(DEV)
    step = runtime.LossStep(weight, b.B, b.L, b.T, DEV, use_graph=True, proj_backward=True)
    step.load(b.hidden, b.links, b.output_length, b.targets, b.target_length)
    stats, mg, lg, loss, d_hidden, d_weight = step.run()
    hid, wt = b.hidden.to(DEV).requires_grad_(True), weight.clone().requires_grad_(True)
    match = ops.proj_logsoftmax_gather_with_grad(hid, wt, b.targets.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV))
    fin = torch.isfinite(match)
    (match[fin] * mg[fin]).sum().backward()
    for got, want in ((d_hidden.float(), hid.grad.float()), (d_weight.float(), wt.grad.float())):
        assert float((got - want).norm() / want.norm()) < 2e-3


@pytest.mark.parametrize("T", [8192, 8200])
def test_projection_with_more_targets_than_are_sorted_in_shared_memory(ops, T):
    """Targets ranked from shared memory and, beyond 8 192, from global memory (ids outside the vocabulary among them): emissions
    against float64 from half-precision operands, float32 sums of 64 products: 1e-4."""
    g = torch.Generator(DEV).manual_seed(T)
    hidden, weight = torch.randn(1, 4, 64, device=DEV, generator=g).half(), (torch.randn(301, 64, device=DEV, generator=g) * 0.2).half()
    targets = torch.randint(0, 301, (1, T), device=DEV, generator=g)
    ops.read_status(DEV)
    got = ops.proj_logsoftmax_gather(hidden, weight, targets, None, None)["match"]
    want = torch.log_softmax(hidden.double() @ weight.double().t(), -1).gather(2, targets[:, None].expand(-1, 4, -1))
    assert (got.double() - want).abs().max() <= 1e-4 and ops.read_status(DEV) == 0
    targets[0, 7], targets[0, T - 1] = 301, -1
    got = ops.proj_logsoftmax_gather(hidden, weight, targets, None, None)["match"]
    assert torch.isnan(got[0, :, [7, T - 1]]).all() and (got[0, :, 8:T - 1].double() - want[0, :, 8:T - 1]).abs().max() <= 1e-4
    assert ops.read_status(DEV) != 0


@pytest.mark.parametrize("V", [33, 513, 1001])
def test_projection_backward_of_an_odd_vocabulary_and_one_row(pkg, ops, V):
    """One real row, as n_rows and as the whole tensor, and a step whose batch has one real node or none; bounds of the test of
    more rows."""
    import importlib
    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    B, L, H, T = 2, 6, 64, 3
    g = torch.Generator(DEV).manual_seed(V)
    hidden, weight = torch.randn(B, L, H, device=DEV, generator=g).half(), (torch.randn(V, H, device=DEV, generator=g) * 0.1).half()
    targets, grad = torch.randint(0, V, (B, T), device=DEV, generator=g), torch.randn(B, L, T, device=DEV, generator=g)
    one = torch.tensor([1, 0], device=DEV)
    cases = [(hidden, targets, grad, one, 1), (hidden[:1, :1], targets[:1], grad[:1, :1], None, None)]
    for hid, tgt, gr, ol, n_rows in cases:
        h64, w64 = hid.double().requires_grad_(), weight.double().requires_grad_()
        lp = torch.log_softmax(h64 @ w64.t(), -1).gather(2, tgt[:, None].expand(-1, hid.shape[1], -1))
        want = torch.autograd.grad((lp * gr)[0, 0].sum(), (h64, w64))
        h, w = hid.clone().requires_grad_(), weight.clone().requires_grad_()
        got = torch.autograd.grad(ops.proj_logsoftmax_gather_with_grad(h, w, tgt, ol, None, n_rows=n_rows), (h, w), gr)
        for x, y in zip(got, want):
            assert (x.double() - y).norm() <= 1e-2 * y.norm() and (x.double() - y).abs().max() <= 3e-2 * y.abs().max()
    step = runtime.LossStep(weight, B, L, T, DEV, use_graph=False, proj_backward=True)
    for real in (1, 0):
        step.load(hidden, torch.full((B, L, 2, L), float("-inf"), device=DEV), real * one, targets, torch.ones(B, dtype=torch.long, device=DEV))
        d_hidden, d_weight = step.run()[-2:]
        assert (d_hidden[1] == 0).all() and (d_hidden[0, real:] == 0).all() and (real or (d_weight == 0).all())
    ops.read_status(DEV)


@pytest.mark.parametrize("n, V, pitch, offset", [(5, 33, 40, 0), (5, 33, 40, 3), (1, 1001, 1008, 1), (4, 999, 999, 0), (3, 64, 64, 0)])
def test_projection_backward_products_of_any_view(ops, n, V, pitch, offset):
    """The public products take d-logits of any V, pitch and offset.  Odd vocabularies go through torch's matmul, which may round
    partial sums and the result to bf16: 2^-9 of each part twice, and a part is no larger than the sum of its terms' magnitudes."""
    g = torch.Generator(DEV).manual_seed(V)
    buffer = torch.randn(offset + n * pitch, device=DEV, generator=g).to(torch.bfloat16)
    dlogits = buffer[offset:].view(n, pitch)[:, :V]
    weight, rows = torch.randn(V, 64, device=DEV, generator=g).half(), torch.randn(n, 64, device=DEV, generator=g).half()
    got = ops.proj_backward_products(dlogits, weight, rows)
    left, right = (dlogits.double(), weight.bfloat16().double()), (dlogits.double().t(), rows.bfloat16().double())
    for x, (a, b) in zip(got, (left, right)):
        assert x.dtype == torch.float32 and ((x.double() - a @ b).abs() <= 2.0 ** -8 * (a.abs() @ b.abs())).all()


@pytest.mark.parametrize("V", [1001, 1007, 2051, 16384, 16387, 33001])
@pytest.mark.parametrize("dtype, offset, columns", [(torch.float16, 0, 20), (torch.float16, 3, 600), (torch.float32, 0, 600),
                                                    (torch.float32, 1, 20)])
def test_logsoftmax_gather_of_unaligned_rows(ops, V, dtype, offset, columns):
    """Rows that start and end between 16-byte boundaries (and bodies of exactly one chunk), more columns than threads, with
    and without the softmax in place, against float64; what lies before and after the rows stays.  Fast exponentials over
    float32 sums of up to 33 001 terms: 1e-5 of a log-probability's scale, 2e-5 of a probability (and a half's rounding)."""
    g = torch.Generator(DEV).manual_seed(V)
    rows = 5
    buffer = torch.randn(offset + rows * V + 64, device=DEV, generator=g).mul_(3).to(dtype)
    buffer[offset + V - 1], buffer[offset + 2 * V] = 30, -60000 if dtype == torch.float16 else float("-inf")
    sel = torch.randint(0, V, (1, rows, columns), device=DEV, generator=g)
    sel[..., 0], sel[..., 1] = 0, V - 1
    x = buffer[offset:offset + rows * V].view(1, rows, V).double()
    want = torch.log_softmax(x, -1)
    for in_place in (True, False):
        mine = buffer.clone()
        assert mine.data_ptr() % 16 == 0
        got = ops.get_pcfg_kernel().logsoftmax_gather(mine[offset:offset + rows * V].view(1, rows, V), sel, in_place)
        picked = want.gather(2, sel)
        finite = torch.isfinite(picked)
        assert torch.equal(torch.isfinite(got), finite)
        assert ((got.double() - picked)[finite].abs() <= 1e-5 * picked[finite].abs().clamp(min=1)).all()
        assert torch.equal(mine[:offset], buffer[:offset]) and torch.equal(mine[offset + rows * V:], buffer[offset + rows * V:])
        after = mine[offset:offset + rows * V].view(1, rows, V)
        if not in_place:
            assert torch.equal(after, buffer[offset:offset + rows * V].view(1, rows, V))
            continue
        p = want.exp()
        bound = 2e-5 * p + (2.0 ** -11 * p + 2.0 ** -24 if dtype == torch.float16 else 1e-38)
        assert ((after.double() - p).abs() <= bound).all()


@pytest.mark.parametrize("V", [2051, 33001])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_logsoftmax_gather_of_unaligned_rows_with_a_large_offset(ops, V, dtype):
    """Logits around 4 000: their differences are exact, so log-probabilities and the softmax are as good as around 0 (a rounded
    product of the largest logit and log2(e) would put 2e-4 on both).  Fast exponentials, float32 sums: 1e-5 of a
    log-probability's scale, 2e-5 of a probability (and a half's rounding)."""
    g = torch.Generator(DEV).manual_seed(V)
    rows, columns = 6, 40
    offset = torch.tensor([0, 999, -4001, 4003, 3999.5, -2500.25], device=DEV)[:, None]
    logits = (torch.randn(rows, V, device=DEV, generator=g) * 3 + offset).to(dtype)[None].contiguous()
    sel = torch.randint(0, V, (1, rows, columns), device=DEV, generator=g)
    want = torch.log_softmax(logits.double(), -1)
    got = ops.get_pcfg_kernel().logsoftmax_gather(logits, sel, True)
    picked, p = want.gather(2, sel), want.exp()
    assert ((got.double() - picked).abs() <= 1e-5 * picked.abs().clamp(min=1)).all()
    bound = 2e-5 * p + (2.0 ** -11 * p + 2.0 ** -24 if dtype == torch.float16 else 1e-38)
    assert ((logits.double() - p).abs() <= bound).all()


def test_copy_real_rows_sends_the_real_nodes_only(ops):
    """pcfgnat_copy_real_rows: rows l < length arrive, the others keep what they held; lengths beyond the tensor
    and below zero are clamped; full sentences next to each other go as one copy; a sentence range."""
    k = ops.get_pcfg_kernel()
    g = torch.Generator().manual_seed(3)
    B, L, H = 7, 12, 40
    src = torch.randn(B, L, H, generator=g).half().pin_memory()
    lengths = torch.tensor([3, 12, 12, 0, 20, -4, 5])
    dst = torch.full((B, L, H), 7.0, dtype=torch.float16, device=DEV)
    assert k.copy_real_rows(dst, src, lengths) == 3 + 12 + 12 + 12 + 5
    torch.cuda.synchronize()
    m = lengths.clamp(0, L)
    for b in range(B):
        assert torch.equal(dst[b, :m[b]].cpu(), src[b, :m[b]])
        assert (dst[b, m[b]:] == 7).all()
    # at most 2 copies: runs are rows [0,3), [12,36), [48,60), [72,77); the gaps of 9 and 12 rows are closed first
    dst.fill_(7.0)
    sent = k.copy_real_rows(dst, src, lengths, max_copies=2)
    torch.cuda.synchronize()
    flat_d, flat_s = dst.view(B * L, H).cpu(), src.view(B * L, H)
    assert sent == 60 + 5 and torch.equal(flat_d[:60], flat_s[:60]) and torch.equal(flat_d[72:77], flat_s[72:77])
    assert (flat_d[60:72] == 7).all() and (flat_d[77:] == 7).all()
    dst.fill_(7.0)
    k.copy_real_rows(dst, src, lengths, 1, 3)
    torch.cuda.synchronize()
    assert torch.equal(dst[1:3].cpu(), src[1:3]) and (dst[0] == 7).all() and (dst[3:] == 7).all()
    with pytest.raises(RuntimeError, match="host"):
        k.copy_real_rows(dst, src, lengths.to(DEV))


def test_fused_projection_flags_bad_targets(ops):
    g = torch.Generator().manual_seed(0)
    hidden = torch.randn(1, 16, 64, generator=g).half().to(DEV)
    weight = torch.randn(300, 64, generator=g).half().to(DEV)
    targets = torch.tensor([[5, 300, 7, -1]], device=DEV)
    ops.read_status(DEV)
    out = ops.proj_logsoftmax_gather(hidden, weight, targets)
    m = out["match"]
    assert torch.isnan(m[0, :, 1]).all() and torch.isnan(m[0, :, 3]).all()
    assert torch.isfinite(m[0, :, 0]).all() and torch.isfinite(m[0, :, 2]).all()
    assert ops.read_status(DEV) & 4
    with pytest.raises(RuntimeError, match="multiple of 64"):
        ops.proj_logsoftmax_gather(hidden[:, :, :48].contiguous(), weight[:, :48].contiguous(), targets)


# ---- the fixed-shape step object (CUDA-graph replay) ---------------------------------------------------------------

def test_loss_step_graph_replay_matches_eager(pkg, ops, syn):
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("step", batch=6, vocab=3000, hidden=128, src_min=5, src_max=20, hidden_std=1.0)
    b1, b2 = syn.make_batch(w, seed=1), syn.make_batch(w, seed=2)
    L, T = max(b1.L, b2.L), max(b1.T, b2.T)

    def padded(b):
        hid = torch.zeros(b.B, L, w.hidden, dtype=torch.float16)
        hid[:, :b.L] = b.hidden
        lk = torch.full((b.B, L, 2, L), float("-inf"))
        lk[:, :b.L, :, :b.L] = b.links
        tg = torch.ones(b.B, T, dtype=torch.long)
        tg[:, :b.T] = b.targets
        return hid, lk, b.output_length, tg, b.target_length  # LossStep.load order

    weight = b1.weight.to(DEV)
    eager = runtime.LossStep(weight, w.batch, L, T, DEV, use_graph=False)
    graphed = runtime.LossStep(weight, w.batch, L, T, DEV, use_graph=True)
    # the graphs are captured on the first batch and replayed on the others; the last two loads go over the
    # copy stream, transitions last, each stage waiting for its own inputs only
    for b, overlap in ((b1, False), (b2, False), (b1, True), (b2, True)):
        args = padded(b)
        eager.load(*args)
        graphed.load(*[t.pin_memory() for t in args], overlap=overlap)
        se, mge, lge, le = [t.clone() for t in eager.run()]
        sg, mgg, lgg, lg_ = graphed.run()
        torch.cuda.synchronize()
        assert torch.isfinite(le).all()
        assert torch.equal(lg_, le) and torch.equal(sg, se)
        assert torch.equal(mgg, mge) and torch.equal(lgg, lge)
        # and against the torch reference of the projection feeding the oracle
        hid, lk, ol, tg, tl = args
        lp = torch.log_softmax(hid.float() @ b1.weight.float().t(), -1)  # the step objects hold b1's projection matrix
        match = lp.gather(2, tg[:, None, :].expand(-1, L, -1)).contiguous()
        syn.eos_mask_(match, ol, tl)
        So, _ = oracle.pcfg_loss(match.numpy(), lk.numpy(), ol.numpy(), tl.numpy())
        np.testing.assert_allclose(le.cpu().numpy(), So[:, 0, 0], rtol=1e-4)
        want = -(torch.from_numpy(So[:, 0, 0]) / tl).sum()
        assert abs(float(-se[0]) - float(want)) < 1e-3 * abs(float(want)) and int(se[1]) == w.batch


def test_empty_and_minimal_inputs(ops, syn):
    k = ops.get_pcfg_kernel()
    L, T = 8, 3
    ma = torch.zeros(0, L, T, device=DEV)
    lk = torch.zeros(0, L, 2, L, device=DEV)
    n0 = torch.zeros(0, dtype=torch.long, device=DEV)
    # no sentences at all: every operator returns empty outputs without launching anything harmful
    S, C = k.pcfg_loss(ma, lk, n0, n0, 1)
    assert S.shape[0] == 0 and C.shape[0] == 0
    loss, mg, lg = k.pcfg_loss_fwd_bwd(ma, lk, n0, n0)
    assert loss.numel() == 0 and mg.shape == ma.shape and lg.shape == lk.shape
    assert k.pcfg_best_tree(S, None, ma, lk, n0, n0, 1).shape == (0, L)
    Sv, R, Lt, Mt = k.pcfg_viterbi(torch.zeros(0, L, device=DEV), lk, n0, 1)
    assert Sv.shape == (0, L, L // 4)
    tok, cnt = k.viterbi_decoding_device(n0, n0, Lt, R, Mt, torch.zeros(0, L, dtype=torch.long, device=DEV),
                                         torch.zeros(L, L, dtype=torch.long, device=DEV), 1)
    assert tok.shape == (0, L) and cnt.numel() == 0
    em = k.proj_logsoftmax_gather(torch.zeros(0, L, 64, dtype=torch.float16, device=DEV),
                                  torch.zeros(100, 64, dtype=torch.float16, device=DEV),
                                  torch.zeros(0, T, dtype=torch.long, device=DEV), n0, n0, want_max=True)
    assert em["match"].shape == (0, L, T) and em["argmax"].shape == (0, L)
    assert k.loss_stats(loss, n0).cpu().tolist() == [0.0, 0.0, 0.0]
    torch.cuda.synchronize()
    # the smallest sentence the grammar admits: two graph nodes... and the smallest table the decoder admits
    b = syn.make_batch(syn.Workload("min", batch=3, vocab=30, hidden=8, src_min=1, src_max=2, emissions="logits"),
                       seed=3)
    ma2 = syn.reference_match_all(b)
    S2, C2 = k.pcfg_loss(ma2.to(DEV), b.links.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV), 1)
    So, Co = oracle.pcfg_loss(ma2.numpy(), b.links.numpy(), b.output_length.numpy(), b.target_length.numpy())
    _rel_close(S2.cpu().numpy(), So, 1e-5, 1e-5)
    tree = k.pcfg_best_tree(S2, None, ma2.to(DEV), b.links.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV), 1)
    want = oracle.pcfg_best_tree(S2.cpu().numpy(), Co, ma2.numpy(), b.links.numpy(), b.output_length.numpy(),
                                 b.target_length.numpy())
    np.testing.assert_array_equal(tree.cpu().numpy(), want)
    assert ops.read_status(DEV) == 0


@pytest.mark.parametrize("L", [12, 9])
def test_copy_links_main_rows(ops, L):
    k = ops.get_pcfg_kernel()
    g = torch.Generator().manual_seed(L)
    src = torch.randn(3, L, 2, L, generator=g)
    for s_ in (src.pin_memory(), src.to(DEV)):
        dst = torch.full((3, L, 2, L), -7.0, device=DEV)
        k.copy_links_main_rows(dst, s_)
        torch.cuda.synchronize()
        assert torch.equal(dst[:, 1::2].cpu(), src[:, 1::2])  # main-chain nodes
        assert (dst[:, 0::2] == -7.0).all()  # rows no kernel reads keep their contents


@pytest.mark.parametrize("B, L, T", [(1, 4, 2), (3, 34, 9), (2, 66, 20), (70, 64, 16), (74, 130, 12), (90, 160, 48),
                                     (80, 262, 20), (150, 96, 11), (8, 514, 100), (5, 640, 30)])
def test_reference_order_table_edges(ops, monkeypatch, B, L, T):
    """The inside table in the reference's order, bit for bit that of the 4-lanes-per-node kernel, at chain lengths
    around the lanes, passes and cluster widths of the kernels that the library picks: one sentence and more than the
    GPU has SMs, cost-ordered shared clusters, odd graph lengths, infinite and NaN entries, a length out of range."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_DP_CLUSTER_SIZE", raising=False)
    g = torch.Generator(DEV).manual_seed(L + B)
    match = torch.randn(B, L, T, device=DEV, generator=g) * 3 - 4
    links = torch.randn(B, L, 2, L, device=DEV, generator=g) * 2 - 5
    match[0, 1, 0], links[0, 1, 0, min(3, L - 1)] = float("-inf"), float("nan")
    links[B // 2, 1:3] = float("-inf")
    ol = torch.randint(2, L + 1, (B,), device=DEV, generator=g)
    tl = torch.randint(1, T + 1, (B,), device=DEV, generator=g)
    ol[-1], tl[-1] = L, T
    if B > 2:
        ol[1] = L + 1
    k = ops.get_pcfg_kernel()
    S, C = k.pcfg_loss(match, links, ol, tl, 1)
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
    S_rows, C_rows = k.pcfg_loss(match, links, ol, tl, 1)
    assert np.array_equal(_bits(S.cpu().numpy()), _bits(S_rows.cpu().numpy()))
    assert np.array_equal(_bits(C.cpu().numpy()), _bits(C_rows.cpu().numpy()))
    assert torch.isfinite(S).any()
    ops.read_status(DEV)


@pytest.mark.parametrize("H", [8, 64, 520, 12])
def test_convert_rows(ops, H):
    """Gather to bf16 and scatter from float32 with the roundings of torch's conversions, with infinities, NaN and
    denormals; a row length that the kernels do not take goes through torch."""
    k = ops.get_pcfg_kernel()
    g = torch.Generator(DEV).manual_seed(H)
    src = torch.randn(301, H, device=DEV, generator=g).half()
    src[5, 0], src[6, 1], src[7, 2], src[8, 3] = float("inf"), float("-inf"), float("nan"), 6e-8
    index = torch.randperm(301, device=DEV, generator=g)[:123]
    bits = lambda t: t.view(torch.int16)  # noqa: E731
    assert torch.equal(bits(k.rows_to_bf16(src)), bits(src.to(torch.bfloat16)))
    assert torch.equal(bits(k.rows_to_bf16(src, index)), bits(src[index].to(torch.bfloat16)))
    grad = torch.randn(123, H, device=DEV, generator=g) * 1e5
    grad[0, 0] = 1e-9
    want = torch.full((301, H), -2.0, dtype=torch.float16, device=DEV)
    got = k.rows_from_f32(grad, want.clone(), index)
    want[index] = grad.half()
    assert torch.equal(bits(got), bits(want))
    assert torch.equal(bits(k.rows_from_f32(grad, torch.zeros(123, H, dtype=torch.float16, device=DEV))), bits(grad.half()))
    assert k.rows_to_bf16(src[:0]).shape == (0, H)


def test_projection_as_the_first_call_of_a_thread(ops):
    """A thread that has made no CUDA call yet (an autograd thread, a server's worker) has no context until one is bound: the
    tensor maps are encoded for it all the same."""
    import threading

    k = ops.get_pcfg_kernel()
    h, w = torch.randn(2, 16, 64, device=DEV).half(), (torch.randn(96, 64, device=DEV) * 0.1).half()
    targets = torch.randint(0, 96, (2, 5), device=DEV)
    out = k.proj_logsoftmax_gather(h, w, targets, want_lse=True)
    grad = torch.randn(2, 16, 5, device=DEV)
    calls = [lambda: k.proj_logsoftmax_gather(h, w, targets)["match"],
             lambda: k.proj_dlogits(h, w, targets, None, None, out["lse"], grad)]
    dl, wb, rows = calls[1](), w.to(torch.bfloat16), h.view(32, 64).to(torch.bfloat16)
    calls.append(lambda: k.proj_backward_gemms(dl, wb, rows)[1])
    for call in calls:
        want, got = call(), []
        torch.cuda.synchronize()
        thread = threading.Thread(target=lambda: got.append(call()))
        thread.start()
        thread.join()
        torch.cuda.synchronize()
        assert len(got) == 1 and torch.equal(got[0], want)


def test_convert_rows_checks_its_index(ops):
    """What torch's index operators converted or refused still is: 32-bit indices, rows that do not match."""
    k = ops.get_pcfg_kernel()
    src = torch.randn(20, 16, device=DEV).half()
    index = torch.tensor([3, 0, 19], device=DEV)
    assert torch.equal(k.rows_to_bf16(src, index.int()), src[index].to(torch.bfloat16))
    dst, grad = torch.zeros(20, 16, dtype=torch.float16, device=DEV), torch.randn(3, 16, device=DEV)
    for args in ((grad, dst, index[:2]), (grad[:, :8].contiguous(), dst, index), (grad, dst, index.int()),
                 (torch.randn(21, 16, device=DEV), dst)):
        with pytest.raises((RuntimeError, IndexError)):
            k.rows_from_f32(*args)
    assert (dst == 0).all()


def test_copy_batch(ops):
    """Tensors of one byte to several blocks, at and off 16- and 4-byte boundaries, the main-chain rows of transitions,
    empty and self copies; overlapping pairs and more pairs than a launch takes are refused with nothing copied."""
    k = ops.get_pcfg_kernel()
    g = torch.Generator(DEV).manual_seed(1)
    pool = torch.randint(0, 256, (1 << 22,), device=DEV, generator=g).to(torch.uint8)
    pairs, at = [], 0
    for size, off in ((1, 0), (15, 0), (4096, 0), (16384 + 16, 0), (100000, 4), (70001, 1), (360, 8), (0, 0), (1 << 20, 0)):
        at = (at + 31) // 16 * 16 + off
        src = pool[at:at + size]
        pairs.append((torch.zeros(size + 16, dtype=torch.uint8, device=DEV)[off:off + size], src))
        at += size
    links = torch.randn(3, 10, 2, 10, device=DEV, generator=g)
    rows = torch.full_like(links, -7.0)
    ids = torch.arange(5, device=DEV)
    assert k.copy_batch(pairs + [(rows, links), (ids, ids)], odd_rows_of=rows)
    for dst, src in pairs:
        assert torch.equal(dst, src)
    assert torch.equal(rows[:, 1::2], links[:, 1::2]) and (rows[:, 0::2] == -7.0).all()
    a, b = torch.zeros(64, device=DEV), torch.ones(64, device=DEV)
    c = b.clone()
    assert not k.copy_batch([(a, c), (c[:32], b[32:])]) and not k.copy_batch([(a, b), (a[8:], b[8:])])
    assert not k.copy_batch([(x, y) for x, y in zip(a.split(2), b.split(2))])
    assert (a == 0).all() and (c == 1).all() and k.copy_batch([])


def test_step_load_from_device_tensors(pkg, ops, syn):
    """Inputs on the device go to a step's buffers in one launch: contiguous ones together with a host tensor, a strided
    one and one of another type, and from the step's own buffers (copies in order)."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    b = syn.make_batch(syn.Workload("dl", batch=3, vocab=300, hidden=64, src_min=4, src_max=9), seed=2)
    args = [b.hidden, b.links, b.output_length, b.targets, b.target_length]
    step = runtime.LossStep(b.weight.to(DEV), b.B, b.L, b.T, DEV)
    step.load(*args)
    want = [t.cpu() for t in step.run()]
    dev = [t.to(DEV) for t in args]
    strided = torch.stack([dev[0], dev[0]], -1)[..., 0]
    for tensors in (dev, [strided, dev[1], args[2], dev[3].int(), dev[4]],
                    [step.hidden, step.links, step.output_length, step.targets, step.target_length]):
        step.load(*tensors)
        for got, ref in zip(step.run(), want):
            assert torch.equal(got.cpu(), ref)
    assert torch.isinf(step.links[:, 0::2]).all()


def test_loss_stats_and_glance_select(ops):
    k = ops.get_pcfg_kernel()
    g = torch.Generator().manual_seed(11)
    loss = -torch.rand(37, generator=g) * 50
    loss[3], loss[20], loss[21] = float("-inf"), float("nan"), float("inf")
    tl = torch.randint(1, 40, (37,), generator=g)
    tl[5] = 0  # clamped to 1
    stats = k.loss_stats(loss.to(DEV), tl.to(DEV)).cpu()
    ok = torch.isfinite(loss)
    want = (loss[ok].double() / tl[ok].clamp(min=1).double()).sum()
    assert abs(float(stats[0]) - float(want)) < 1e-5 * abs(float(want))
    assert stats[1] == 37 and stats[2] == 3
    assert k.loss_stats(loss[:0].to(DEV), tl[:0].to(DEV)).cpu().tolist() == [0.0, 0.0, 0.0]

    for B, L, T, p, seed in ((5, 40, 12, 0.5, 0), (3, 300, 90, 0.3, 1), (2, 16, 5, 1.0, 2), (4, 24, 7, 0.0, 3)):
        g = torch.Generator().manual_seed(seed)
        tlen = torch.randint(2, T + 1, (B,), generator=g)
        path = torch.randint(-1, T + 2, (B, L), generator=g)  # also positions past the target (dropped from the mask)
        path[torch.rand(B, L, generator=g) < 0.4] = -1
        tgt = torch.randint(4, 50, (B, T), generator=g)
        pred = torch.randint(4, 50, (B, L), generator=g)
        pred = torch.where(torch.rand(B, L, generator=g) < 0.5, tgt.gather(-1, path.clip(0, T - 1)), pred)
        prev = torch.randint(1, 4, (B, L), generator=g)
        noise = torch.randn(B, L, generator=g)
        noise[0, : L // 2] = noise[0, 0]  # ties at the threshold
        got = k.glance_select(path.to(DEV), pred.to(DEV), tgt.to(DEV), prev.to(DEV), tlen.to(DEV), noise.to(DEV), p)
        want = pyref.glance_select(path, pred, tgt, prev, tlen, noise, p)
        for key, val in want.items():
            assert torch.equal(got[key].cpu(), val), (key, B, L, T)


@pytest.mark.parametrize("B, L, T", [(1, 2, 1), (3, 41, 12), (2, 255, 33), (2, 256, 31), (4, 130, 64), (2, 1030, 40), (1, 29500, 3)])
@pytest.mark.parametrize("strategy", ["number-random", "cmlm", None])
def test_glance_select_sizes(ops, B, L, T, strategy):
    """Rows of the match mask in words and in bytes, more nodes than threads, and graphs whose alignment has no room in shared
    memory: every output against the torch restatement (positions past the target and ties included)."""
    g = torch.Generator().manual_seed(L)
    tlen = torch.randint(1, T + 1, (B,), generator=g)
    path = torch.randint(-1, T + 2, (B, L), generator=g)
    path[torch.rand(B, L, generator=g) < 0.4] = -1
    tgt, pred = torch.randint(4, 9, (B, T), generator=g), torch.randint(4, 9, (B, L), generator=g)
    prev = torch.randint(1, 4, (B, L), generator=g)
    noise = torch.randn(B, L, generator=g)
    noise[:, ::3] = noise[:, :1].clone()
    uniform = torch.rand((B, L) if strategy is None else (B,), generator=g)
    k = ops.get_pcfg_kernel()
    d = lambda t: t.to(DEV)  # noqa: E731
    got = k.glance_select(d(path), d(pred), d(tgt), d(prev), d(tlen), d(noise), 0.5, strategy, d(uniform))
    want = pyref.glance_select(path, pred, tgt, prev, tlen, noise, 0.5, strategy, uniform)
    for key, val in want.items():
        assert torch.equal(got[key].cpu(), val), key


def test_glance_select_just_below_48_kb_of_shared_memory():
    """6 140 nodes ask for 49 120 bytes beside the kernel's own 128, in a process of their own: an earlier call for a longer graph
    raises the kernel's limit for good."""
    import subprocess
    import sys

    from conftest import ROOT

    program = """
import sys; sys.path.insert(0, "tests")
import torch, _pyref as pyref, __graft_entry__ as entry
entry.load_package()
from pcfg_nat_b200.custom_ops import pcfg_loss as ops
B, L, T = 2, 6140, 3
g = torch.Generator().manual_seed(1)
args = [torch.randint(-1, T, (B, L), generator=g), torch.randint(4, 9, (B, L), generator=g), torch.randint(4, 9, (B, T), generator=g),
        torch.ones(B, L, dtype=torch.long), torch.tensor([3, 2]), torch.randn(B, L, generator=g)]
got = ops.get_pcfg_kernel().glance_select(*[t.cuda() for t in args], 0.5, "number-random", None)
for key, val in pyref.glance_select(*args, 0.5, "number-random", None).items():
    assert torch.equal(got[key].cpu(), val), key
"""
    r = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("case", ["small", "mid"])
def test_extract_links_against_reference_model(ops, case):
    """links from the projected link features against the reference model's own extract_links (run on the CPU
    by tests/golden/make_golden_links.py)."""
    g = np.load(golden_path("host_extract_links.npz"))
    heads = int(g[f"{case}_heads"])
    q, kl, kr = (torch.from_numpy(g[f"{case}_{n}"]) for n in ("q", "kl", "kr"))
    B, L, E = q.shape
    shape = (B, L, heads, E // heads)
    links = ops.get_pcfg_kernel().extract_links(
        q.view(shape).to(DEV), kl.view(shape).to(DEV), kr.view(shape).to(DEV), torch.from_numpy(g[f"{case}_gates"]).to(DEV),
        torch.from_numpy(g[f"{case}_prev"]).to(DEV), 1, torch.from_numpy(g[f"{case}_left_mask"]),
        torch.from_numpy(g[f"{case}_right_mask"]), torch.from_numpy(g[f"{case}_main_chain"]))
    want = g[f"{case}_links"]
    got = links.cpu().numpy()
    assert got.shape == want.shape
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    fin = np.isfinite(want)
    assert fin.sum() > 20
    np.testing.assert_allclose(got[fin], want[fin], rtol=1e-4, atol=1e-5)
    # the rows of a node are a distribution over (left option, right child)
    rows = np.isfinite(want).any(axis=(2, 3))
    mass = np.exp(got[rows].reshape(rows.sum(), -1).astype(np.float64)).sum(-1)
    np.testing.assert_allclose(mass, 1.0, atol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("case", ["small", "mid"])
def test_extract_links_backward_against_reference_autograd(ops, case, dtype):
    """The hand-written backward of extract_links against the reference model's own function differentiated by
    autograd (tests/golden/make_golden_links.py): gradient of sum(links * G) over the finite entries with respect to
    the three link feature tensors and the gate logits."""
    g = np.load(golden_path("host_extract_links.npz"))
    heads = int(g[f"{case}_heads"])
    t = lambda n: torch.from_numpy(g[f"{case}_{n}"])
    B, L, E = t("q").shape
    shape = (B, L, heads, E // heads)
    leaves = [t(n).view(shape).to(DEV, dtype).requires_grad_(True) for n in ("q", "kl", "kr")]
    gates = t("gates").to(DEV).requires_grad_(True)
    links = ops.get_pcfg_kernel().extract_links(*leaves, gates, t("prev").to(DEV), 1, t("left_mask"), t("right_mask"),
                                                t("main_chain"))
    assert links.requires_grad
    fin = torch.isfinite(links)
    (torch.where(fin, links, torch.zeros_like(links)) * t("G").to(DEV)).sum().backward()
    tol = dict(rtol=1e-3, atol=1e-5) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)  # f16 inputs are rounded
    for leaf, name in zip(leaves, ("dq", "dkl", "dkr")):
        assert leaf.grad.dtype == dtype
        np.testing.assert_allclose(leaf.grad.float().cpu().numpy().reshape(B, L, E), g[f"{case}_{name}"], **tol)
    np.testing.assert_allclose(gates.grad.cpu().numpy(), g[f"{case}_dgates"], **tol)
    if dtype == torch.float32:  # and through the loss: d loss / d link features, against float64 torch autograd
        import importlib

        match = torch.randn(B, L, 5, device=DEV).log_softmax(0)
        ol = t("prev").ne(1).sum(1).to(DEV)
        tl = torch.full((B,), 5, device=DEV)
        for x in leaves + [gates]:
            x.grad = None
        links = ops.get_pcfg_kernel().extract_links(*leaves, gates, t("prev").to(DEV), 1, t("left_mask"), t("right_mask"),
                                                    t("main_chain"))
        loss = ops.cuda_pcfg_loss(match, links, ol, tl)
        ok = torch.isfinite(loss)
        assert ok.any()
        loss[ok].sum().backward()
        assert all(torch.isfinite(x.grad).all() for x in leaves + [gates]) and leaves[0].grad.abs().sum() > 0


@pytest.mark.parametrize("L, heads, dim, dtype", [(2, 1, 4, torch.float32), (9, 3, 5, torch.float32), (62, 1, 33, torch.float16),
                                                  (64, 4, 64, torch.float16), (66, 2, 68, torch.float32),
                                                  (128, 8, 16, torch.float16), (131, 5, 64, torch.float16),
                                                  (322, 8, 64, torch.float16)])
def test_extract_links_and_gradient_at_tile_edges(pkg, ops, L, heads, dim, dtype):
    """Transitions and feature gradients at node and feature counts around the tiles of the product kernels, against
    autograd in float64: float32 sums of up to 322 terms, 2e-5 of the largest entry (half precision: its rounding)."""
    import importlib

    lm, rm, mc = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)
    g = torch.Generator().manual_seed(L)
    leaves = [torch.randn(3, L, heads, dim, generator=g).to(dtype) for _ in range(3)] + [torch.randn(3, L, heads, generator=g)]
    length = torch.tensor([L, max(2, L // 2), max(2, L - 3)])
    prev = torch.where(torch.arange(L)[None, :] < length[:, None], 3, 1)
    ref = [t.double().requires_grad_() for t in leaves]
    want = pyref.extract_links(*ref, prev, 1, lm, rm, mc, dtype=torch.float64, floor=-1e30)
    ours = [t.to(DEV).requires_grad_() for t in leaves]
    links = ops.get_pcfg_kernel().extract_links(*ours, prev.to(DEV), 1, lm, rm, mc)
    ok = want > -1e29
    assert torch.equal(torch.isfinite(links).cpu(), ok)
    G = torch.randn(want.shape, generator=g) * ok
    torch.testing.assert_close(links.detach().cpu()[ok].double(), want.detach()[ok], rtol=1e-5, atol=1e-4)
    if not ok.any():
        return
    torch.where(ok, want, 0.0).mul(G).sum().backward()
    (torch.where(ok.to(DEV), links, 0.0) * G.to(DEV)).sum().backward()
    for x, y in zip(ours, ref):
        err = (x.grad.cpu().double() - y.grad).abs().max()
        assert err <= (2e-5 if x.dtype == torch.float32 else 1e-3) * y.grad.abs().max(), (tuple(x.shape), float(err))


def test_extract_links_under_inference_mode(pkg, ops):
    """Inference tensors have no version counter: masks made inside the mode (bool or host masks are converted there)
    work, one that is changed in place there is read again, and a mask from outside the mode works in it."""
    import importlib

    L, heads, dim = 18, 2, 8
    masks = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)
    g = torch.Generator().manual_seed(3)
    feats = [torch.randn(2, L, heads, dim, generator=g).to(DEV) for _ in range(3)] + [torch.randn(2, L, heads, generator=g).to(DEV)]
    prev = torch.full((2, L), 3, device=DEV)
    u8 = [m.to(DEV).ne(0).to(torch.uint8) for m in masks]
    k = ops.get_pcfg_kernel()
    want = k.extract_links(*feats, prev, 1, *u8)
    shorter = u8[2].clone()
    shorter[L - 3:] = 0
    want_shorter = k.extract_links(*feats, prev, 1, u8[0], u8[1], shorter)
    assert not torch.equal(want, want_shorter)
    with torch.inference_mode():
        inside = [m.to(DEV).ne(0).to(torch.uint8) for m in masks]
        for given in ([m.bool() for m in masks], [m.to(DEV).bool() for m in masks], u8, inside):
            assert torch.equal(k.extract_links(*feats, prev, 1, *given), want)
        inside[2][L - 3:] = 0
        assert torch.equal(k.extract_links(*feats, prev, 1, *inside), want_shorter)


def test_extract_links_on_another_stream_than_the_first(pkg, ops):
    """The node lists that a mask's first call leaves for later ones: a call on another stream reads them when its turn
    comes, also if a call with another mask has taken their place and their memory was handed out again by then."""
    import importlib

    get_mask, k = importlib.import_module("pcfg_nat_b200.support_tree").get_mask, ops.get_pcfg_kernel()
    g = torch.Generator(DEV).manual_seed(4)

    def inputs(L):
        masks = [m.to(DEV).ne(0).to(torch.uint8) for m in get_mask(L, 1)]
        feats = [torch.randn(2, L, 2, 8, device=DEV, generator=g) for _ in range(3)]
        return [*feats, torch.randn(2, L, 2, device=DEV, generator=g), torch.full((2, L), 3, device=DEV), 1, *masks]

    first, second = inputs(60), inputs(30)
    want = k.extract_links(*first)
    side = torch.cuda.Stream(DEV)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)  # a tenth of a second
        got = k.extract_links(*first)
    k.extract_links(*second)
    filler = [torch.zeros(n, dtype=torch.int32, device=DEV) for n in (30, 60) for _ in range(64)]
    torch.cuda.synchronize()
    assert torch.equal(got, want), len(filler)


def _tree_masks(L):
    import importlib

    return [m.to(DEV) for m in importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)]


def _links_and_float64(pkg, ops, leaves, length, G_of):
    """(links, gradients of the leaves, both again by autograd in float64): G_of(float64 links) weighs the finite cells."""
    import importlib

    L = leaves[0].shape[1]
    masks = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)
    prev = torch.where(torch.arange(L)[None, :] < length[:, None], 3, 1)
    ref = [t.double().requires_grad_() for t in leaves]
    want = pyref.extract_links(*ref, prev, 1, *masks, dtype=torch.float64, floor=-1e30)
    ok = want > -1e29
    G = G_of(want.detach()).float() * ok
    torch.where(ok, want, 0.0).mul(G).sum().backward()
    ours = [t.to(DEV).requires_grad_() for t in leaves]
    links = ops.get_pcfg_kernel().extract_links(*ours, prev.to(DEV), 1, *masks)
    (torch.where(ok.to(DEV), links, 0.0) * G.to(DEV)).sum().backward()
    assert torch.equal(torch.isfinite(links).cpu(), ok)
    return links.detach().cpu().double()[ok], [t.grad.cpu().double() for t in ours], want.detach()[ok], [t.grad for t in ref]


@pytest.mark.parametrize("heads", [1, 2])
def test_links_gradient_of_improbable_cells_with_large_weights(pkg, ops, heads):
    """Gradients of 1e12 at transitions of e-69 to e-61, where gradient / probability leaves the floats.  Logits of up to 100
    in float32 (spacing 8e-6, a handful of roundings) put 1e-4 on a probability."""
    g = torch.Generator().manual_seed(heads)
    leaves = [4 * torch.randn(2, 40, heads, 8, generator=g) for _ in range(3)] + [torch.randn(2, 40, heads, generator=g)]
    weights = lambda want: torch.where((want > -69) & (want < -61), 1e12, 0.0)  # noqa: E731
    got, grads, want, ref = _links_and_float64(pkg, ops, leaves, torch.tensor([40, 31]), weights)
    assert int((weights(want) > 0).sum()) > 3
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4)
    for x, y in zip(grads, ref):
        assert (x - y).abs().max() <= 1e-4 * y.abs().max(), tuple(x.shape)


@pytest.mark.parametrize("B, L, heads, dim", [(3, 6, 3, 64), (2, 32, 2, 68), (2, 34, 2, 33), (40, 66, 4, 36), (20, 130, 8, 8)])
def test_links_and_gradient_at_other_tiles(pkg, ops, B, L, heads, dim):
    """The smaller tiles of the product kernels (up to 16, 32 and 31 nodes, and grids smaller than the GPU) and the larger
    one with a single tile of rows, ragged sentences, against float64: float32 sums, 2e-5 of the largest entry."""
    g = torch.Generator().manual_seed(L)
    leaves = [torch.randn(B, L, heads, dim, generator=g) for _ in range(3)] + [torch.randn(B, L, heads, generator=g)]
    length = torch.randint(2, L + 1, (B,), generator=g)
    length[0] = L
    got, grads, want, ref = _links_and_float64(pkg, ops, leaves, length, lambda want: torch.randn(want.shape, generator=g))
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4)
    for x, y in zip(grads, ref):
        assert (x - y).abs().max() <= 2e-5 * y.abs().max(), tuple(x.shape)


@pytest.mark.parametrize("B, L, heads, dim, scale", [(2, 2, 1, 64, 1.0), (3, 3, 3, 32, 1.0), (2, 30, 9, 64, 1.0), (3, 32, 8, 64, 1.0),
                                                     (2, 34, 32, 32, 1.0), (5, 66, 2, 64, 1.0), (1, 95, 12, 64, 1.0),
                                                     (20, 130, 5, 32, 1.0), (64, 98, 1, 64, 1.0), (4, 94, 2, 64, 16.0)])
def test_links_from_half_features_in_registers(pkg, ops, B, L, heads, dim, scale):
    """The kernels without score matrices: chains of 1 to 65 nodes around their tiles of 16, more and fewer heads than a
    block has warps, both head sizes, ragged sentences, improbable cells (scale 16: logits of up to 150 in units of log 2, spacing
    1.5e-5, a handful of roundings: 2e-4), against autograd in float64: float32 sums, 2e-5 of the largest entry before
    the gradients are rounded to half precision (2^-11 of each)."""
    g = torch.Generator().manual_seed(L)
    leaves = [(scale ** 0.5 * torch.randn(B, L, heads, dim, generator=g)).half() for _ in range(3)] + [torch.randn(B, L, heads, generator=g)]
    length = torch.randint(2, L + 1, (B,), generator=g)
    length[0] = L
    k = ops.get_pcfg_kernel()
    kept = k._links_forward(*[t.to(DEV) for t in leaves], torch.full((B, L), 3, device=DEV), 1, *_tree_masks(L))[1]
    assert "kept" in kept  # the kernels under test
    got, grads, want, ref = _links_and_float64(pkg, ops, leaves, length, lambda want: torch.randn(want.shape, generator=g))
    assert scale == 1.0 or int((want < -69.1).sum()) > 3
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4 if scale == 1.0 else 2e-4)
    for x, y, leaf in zip(grads, ref, leaves):
        bound = (2e-5 if scale == 1.0 else 2e-4) * y.abs().max() + (y.abs() * 2.0 ** -11 if leaf.dtype == torch.float16 else 0)
        assert ((x - y).abs() <= bound).all(), tuple(x.shape)


def test_links_from_half_features_by_masks_and_odd_values(pkg, ops):
    """Masks that are no tree's (random left and right children, an irregular main chain) with pads in the middle, features
    with an infinity and a NaN, gradients of 1e12 and 1e-20: the kernels in registers against the ones over float32 scores,
    which take the same features in float32 (sums of up to 40 terms in another order: 2e-5; a half's rounding)."""
    B, L, heads, dim = 3, 44, 3, 32
    g = torch.Generator().manual_seed(5)
    left, right = (torch.rand(L, L, generator=g) < 0.5).to(torch.uint8), (torch.rand(L, L, generator=g) < 0.4).to(torch.uint8)
    chain = (torch.rand(L, generator=g) < 0.8).to(torch.uint8)
    left[:, 0], left[7] = 0, 1
    prev = torch.where(torch.rand(B, L, generator=g) < 0.9, 3, 1)
    prev[:, 0] = 3
    feats = [torch.randn(B, L, heads, dim, generator=g).half() for _ in range(3)] + [torch.randn(B, L, heads, generator=g)]
    feats[0][1, int(chain.nonzero()[5]), 1, 0], feats[2][2, int(chain.nonzero()[9]), 2, 3] = float("inf"), float("nan")
    G = torch.randn(B, L, 2, L, generator=g)
    G[0, :20] *= 1e12
    G[0, 20:] *= 1e-20
    masks = [m.to(DEV) for m in (left, right, chain)]
    k = ops.get_pcfg_kernel()
    half, kept = k._links_forward(*[t.to(DEV) for t in feats], prev.to(DEV), 1, *masks)
    full, saved = k._links_forward(*[t.float().to(DEV) for t in feats], prev.to(DEV), 1, *masks)
    assert "kept" in kept and "kept" not in saved
    assert torch.equal(torch.isfinite(half), torch.isfinite(full))
    torch.testing.assert_close(half, full, rtol=1e-5, atol=1e-4, equal_nan=True)
    G = torch.where(torch.isfinite(full), G.to(DEV), 0)
    for x, y in zip(k._links_backward(G, kept), k._links_backward(G, saved)):
        assert torch.equal(torch.isfinite(x), torch.isfinite(y))
        for b in range(B):  # sentences have scales of their own
            part, of = x[b][torch.isfinite(y[b])], y[b][torch.isfinite(y[b])]
            assert ((part - of).abs() <= 2e-5 * of.abs().max()).all(), (b, tuple(x.shape))


@pytest.mark.parametrize("B, L, heads, dim, by", [(4, 66, 3, 64, "rows"), (4, 66, 3, 64, "cells"), (33, 98, 2, 32, "rows"), (3, 34, 9, 64, "rows")])
def test_links_gradient_of_rows_of_different_sizes(pkg, ops, B, L, heads, dim, by):
    """links_grad rows (or cells) that are up to 1e24 apart, some 1e-12 and less: the feature gradients of every (node, head) against
    autograd in float64, by that row's own size.  Logits of up to 16 in units of log 2 (spacing 2e-6, a handful of roundings) put
    1e-5 on a probability; what a row's cells cancel of one another, two digits at most: 1e-3."""
    g = torch.Generator().manual_seed(L)
    leaves = [torch.randn(B, L, heads, dim, generator=g).half() for _ in range(3)] + [torch.randn(B, L, heads, generator=g)]
    length = torch.randint(L // 2, L + 1, (B,), generator=g)
    length[0] = L
    prev = torch.where(torch.arange(L)[None, :] < length[:, None], 3, 1)
    masks = _tree_masks(L)
    ref = [t.double().requires_grad_() for t in leaves]
    want = pyref.extract_links(*ref, prev, 1, *[m.cpu() for m in masks], dtype=torch.float64, floor=-1e30)
    ok = want > -1e29
    size = torch.rand((B, L, 1, 1) if by == "rows" else (B, L, 2, L), generator=g)
    G = torch.randn(B, L, 2, L, generator=g) * ok * 10 ** (24 * size - 12)
    torch.where(ok, want, 0.0).mul(G).sum().backward()
    k = ops.get_pcfg_kernel()
    _, saved = k._links_forward(*[t.to(DEV) for t in leaves], prev.to(DEV), 1, *[m.ne(0).to(torch.uint8) for m in masks])
    assert "kept" in saved  # the kernels under test
    for got, leaf in zip(k._links_backward(G.to(DEV), saved), ref[:3]):
        got, y = got.cpu().double(), leaf.grad
        assert ((got - y).norm(dim=-1) <= 1e-3 * y.norm(dim=-1)).all()


@pytest.mark.parametrize("heads, scale", [(1, 4.0), (2, 4.0), (8, 5.0)])
def test_links_of_improbable_cells(pkg, ops, heads, scale):
    """Transitions below the probability (1e-30) under which the mixture is formed from log-probabilities, and their
    gradient.  Logits of up to 150 in float32 (spacing 1.5e-5, a handful of roundings): 1e-4."""
    g = torch.Generator().manual_seed(heads)
    leaves = [scale * torch.randn(2, 40, heads, 8, generator=g) for _ in range(3)] + [torch.randn(2, 40, heads, generator=g)]
    got, grads, want, ref = _links_and_float64(pkg, ops, leaves, torch.tensor([40, 31]),
                                               lambda want: torch.randn(want.shape, generator=g))
    assert int((want < -69.1).sum()) > 3
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4)
    for x, y in zip(grads, ref):
        assert (x - y).abs().max() <= 1e-4 * y.abs().max(), tuple(x.shape)


def test_links_with_rows_beyond_shared_memory(pkg, ops):
    """Rows whose exponentials (32 heads x 162 nodes), and rows whose weights (3 725 nodes) stay out of shared memory: the
    same transitions and gradients, against float64.  The long graph's sentences fill its first nodes only, so that it
    has to give what a short graph gives."""
    import importlib

    g = torch.Generator().manual_seed(7)
    leaves = [torch.randn(1, 324, 32, 4, generator=g) for _ in range(3)] + [torch.randn(1, 324, 32, generator=g)]
    got, grads, want, ref = _links_and_float64(pkg, ops, leaves, torch.tensor([324]),
                                               lambda want: torch.randn(want.shape, generator=g))
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4)
    for x, y in zip(grads, ref):
        assert (x - y).abs().max() <= 2e-5 * y.abs().max(), tuple(x.shape)

    L, short, heads = 7450, 140, 2
    masks = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)
    masks = [m.to(DEV).ne(0).to(torch.uint8) for m in masks]
    leaves = [torch.randn(2, short, heads, 8, generator=g) for _ in range(3)] + [torch.randn(2, short, heads, generator=g)]
    length = torch.tensor([short, 77])
    G = torch.randn(2, short, 2, short, generator=g)
    got, grads, want, ref = _links_and_float64(pkg, ops, leaves, length, lambda want: G)
    padded = [torch.cat([t, torch.zeros(2, L - short, *t.shape[2:])], 1).to(DEV).requires_grad_() for t in leaves]
    prev = torch.where(torch.arange(L)[None, :] < length[:, None], 3, 1).to(DEV)
    links = ops.get_pcfg_kernel().extract_links(*padded, prev, 1, *masks)
    part = links[:, :short, :, :short]
    finite = torch.isfinite(part)
    assert int(torch.isfinite(links).sum()) == int(finite.sum())
    torch.testing.assert_close(part.detach()[finite].cpu().double(), want, rtol=1e-5, atol=1e-4)
    (torch.where(finite, part, 0.0) * G.to(DEV)).sum().backward()
    for x, y in zip(padded, ref):
        assert (x.grad[:, :short].cpu().double() - y).abs().max() <= 2e-5 * y.abs().max(), tuple(x.shape)
        assert (x.grad[:, short:] == 0).all()


def test_links_with_an_infinite_logit(pkg, ops):
    """A head with a logit of +inf counts nothing in its row; the others keep their part and their gradients."""
    import importlib

    L, heads, dim = 20, 2, 4
    masks = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)
    g = torch.Generator().manual_seed(2)
    leaves = [torch.randn(1, L, heads, dim, generator=g) for _ in range(3)] + [torch.randn(1, L, heads, generator=g)]
    leaves[0][0, 3, 0], leaves[2][0, 7, 0] = 1e20, 1e20  # node 3, child 7: the product of head 0 is +inf
    ours = [t.to(DEV).requires_grad_() for t in leaves]
    links = ops.get_pcfg_kernel().extract_links(*ours, torch.full((1, L), 3, device=DEV), 1, *masks)
    ref = [t[..., 1:, :].double().requires_grad_() for t in leaves[:3]] + [torch.zeros(1, L, 1).double()]
    want = pyref.extract_links(*ref, torch.full((1, L), 3), 1, *masks, dtype=torch.float64, floor=-1e30)[0, 3]
    ok = want > -1e29
    want = want + torch.log_softmax(leaves[3][0, 3].double(), 0)[1]
    assert torch.equal(torch.isfinite(links[0, 3]).cpu(), ok)
    torch.testing.assert_close(links[0, 3].detach().cpu()[ok].double(), want.detach()[ok], rtol=1e-5, atol=1e-5)
    G = torch.randn(2, L, generator=g) * ok
    (torch.where(ok, want, 0.0) * G).sum().backward()
    (torch.where(ok.to(DEV), links[0, 3], 0.0) * G.to(DEV)).sum().backward()
    for x, y in zip(ours[:3], ref[:3]):
        err = (x.grad[..., 1:, :].cpu().double() - y.grad).abs().max()
        assert err <= 2e-5 * y.grad.abs().max(), (tuple(x.shape), float(err))


def test_links_gradient_of_many_sentences(ops):
    """More (sentence, head) pairs than a grid's second or third dimension takes: the sentences repeat, and so do their
    transitions and gradients."""
    import importlib

    B, L, heads, dim, few = 16400, 4, 4, 4, 50
    masks = [m.to(DEV) for m in importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)]
    g = torch.Generator(DEV).manual_seed(1)
    base = [torch.randn(few, L, heads, dim, device=DEV, generator=g) for _ in range(3)] + \
        [torch.randn(few, L, heads, device=DEV, generator=g)]
    G = torch.randn(few, L, 2, L, device=DEV, generator=g)
    k = ops.get_pcfg_kernel()

    def chain(n):
        leaves = [t.repeat(n, *[1] * (t.dim() - 1)).requires_grad_() for t in base]
        links = k.extract_links(*leaves, torch.full((n * few, L), 3, device=DEV), 1, *masks)
        loss = (torch.where(torch.isfinite(links), links, 0.0) * G.repeat(n, 1, 1, 1)).sum()
        return torch.autograd.grad(loss, leaves)

    for one, many in zip(chain(1), chain(B // few)):
        assert torch.equal(many, one.repeat(B // few, *[1] * (one.dim() - 1))) and one.abs().sum() > 0


def test_decode_step_from_link_features(pkg, ops, syn):
    """DecodeStep fed with the projected link features gives what extract_links + the transition-fed step give."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    support_tree = importlib.import_module("pcfg_nat_b200.support_tree")
    w = syn.Workload("decf", batch=4, vocab=500, hidden=64, src_min=4, src_max=12, kind="viterbi")
    b = syn.make_batch(w, seed=8)
    heads, dim = 8, 16
    g = torch.Generator().manual_seed(3)
    q, kl, kr = (torch.randn(b.B, b.L, heads, dim, generator=g).half() for _ in range(3))
    gates = torch.randn(b.B, b.L, heads, generator=g)
    prev = torch.where(torch.arange(b.L)[None, :] < b.output_length[:, None], 3, 1)
    lm, rm, mc = support_tree.get_mask(b.L, 1)
    k = ops.get_pcfg_kernel()
    links = k.extract_links(q.to(DEV), kl.to(DEV), kr.to(DEV), gates.to(DEV), prev.to(DEV), 1, lm, rm, mc)
    want = pyref.extract_links(q, kl, kr, gates, prev, 1, lm, rm, mc)
    assert torch.equal(torch.isfinite(links).cpu(), torch.isfinite(want))
    fin = torch.isfinite(want)
    torch.testing.assert_close(links.cpu()[fin], want[fin], rtol=1e-4, atol=1e-5)
    weight = b.weight.to(DEV)
    plain = runtime.DecodeStep(weight, b.B, b.L, lm, DEV)
    plain.load(b.hidden.pin_memory(), links, b.output_length.pin_memory())
    feat = runtime.DecodeStep(weight, b.B, b.L, lm, DEV, link_features=(heads, dim), right_tree_mask=rm, main_chain=mc)
    feat.load(b.hidden.pin_memory(), q.pin_memory(), kl.pin_memory(), kr.pin_memory(), gates.pin_memory(),
              prev.pin_memory(), b.output_length.pin_memory(), overlap=True)
    for _ in range(2):
        t1, c1, p1 = [t.clone() for t in plain.run()]
        t2, c2, p2 = [t.clone() for t in feat.run()]
    assert torch.equal(t1, t2) and torch.equal(c1, c2) and torch.equal(p1, p2)
    assert int(c1.min()) >= 1


def test_loss_stats_exchange_bounded_wait(ops):
    """The in-kernel exchange of the loss statistics with a peer that never arrives: the wait runs out, the
    status word says so, the statistics are NaN (never a short sum that could pass for a loss), the host-side
    check raises, and the context stays usable."""
    k = ops.get_pcfg_kernel()
    bufs = [torch.zeros(64, dtype=torch.float32, device=DEV) for _ in range(2)]  # >= PCFGNAT_EXCHANGE_BYTES(2)
    peers = torch.tensor([b.data_ptr() for b in bufs], dtype=torch.int64, device=DEV)
    loss = torch.tensor([-4.0, -9.0, float("-inf")], device=DEV)
    tl = torch.tensor([2, 3, 5], device=DEV)
    ops.read_status(DEV)
    stats = k.loss_stats_exchange(loss, tl, peers, 0, 2).cpu()
    assert torch.isnan(stats).all()
    assert ops.read_status(DEV) & 8  # PCFGNAT_STATUS_TIMEOUT
    import importlib

    sharding = importlib.import_module("pcfg_nat_b200.sharding")
    with pytest.raises(RuntimeError, match="did not arrive"):
        sharding.check_exchanged_stats(stats)
    assert sharding.check_exchanged_stats(torch.tensor([-5.0, 3.0, 1.0])) is None
    # a world of one rank needs nobody else
    one = torch.zeros(64, dtype=torch.float32, device=DEV)
    stats = k.loss_stats_exchange(loss, tl, torch.tensor([one.data_ptr()], dtype=torch.int64, device=DEV), 0, 1).cpu()
    assert stats.tolist() == [-5.0, 3.0, 1.0] and ops.read_status(DEV) == 0


def test_decode_and_glance_steps_match_operator_chain(pkg, ops, syn):
    """The graph-replayed decode / glancing steps give what the individual operators give."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("dec", batch=5, vocab=2000, hidden=64, src_min=6, src_max=24, kind="viterbi")
    b = syn.make_batch(w, seed=4)
    weight = b.weight.to(DEV)
    dec = runtime.DecodeStep(weight, b.B, b.L, b.left_tree_mask, DEV, beta=1.0, pad_index=1)
    dec.load(b.hidden.pin_memory(), b.links.pin_memory(), b.output_length.pin_memory())
    for _ in range(2):  # capture, then replay
        tokens, count, pred = [t.clone() for t in dec.run()]
    torch.cuda.synchronize()
    # reference chain on the CPU: fp32 projection -> log-softmax max -> oracle Viterbi -> oracle back-trace
    lp = torch.log_softmax(b.hidden.float() @ b.weight.float().t(), -1)
    ob, tok = lp.max(-1)
    out = ops.proj_logsoftmax_gather(b.hidden.to(DEV), weight, None, b.output_length.to(DEV), None, want_max=True)
    real = torch.arange(b.L)[None, :] < b.output_length[:, None]
    torch.testing.assert_close(out["max_lprob"].cpu()[real], ob[real], rtol=0, atol=2e-3)
    # Viterbi on the kernel's own emissions (bit-exact path), compared with the oracle on the same numbers
    ob_k, tok_k = out["max_lprob"].cpu(), out["argmax"].cpu()
    So, Ro, Lo, Mo = oracle.pcfg_viterbi(ob_k.numpy(), b.links.numpy(), b.output_length.numpy())
    sc = torch.from_numpy(So[:, 1, :]) / torch.arange(b.L // 4).unsqueeze(0)
    sc = torch.where(torch.isnan(sc), torch.full_like(sc, float("-inf")), sc)
    want_pred = sc[:, 1:].max(-1)[1] + 1
    assert torch.equal(pred.cpu(), want_pred)
    want = oracle.viterbi_decoding_lists(want_pred.numpy(), b.output_length.numpy(), Lo, Ro, Mo, tok_k.numpy(),
                                         b.left_tree_mask.long().numpy(), 1)
    for i, row in enumerate(want):
        assert tokens[i, :int(count[i])].cpu().tolist() == row
        assert (tokens[i, int(count[i]):] == 1).all()

    wg = syn.Workload("gl", batch=4, vocab=2000, hidden=64, src_min=6, src_max=20, kind="glance")
    g = syn.make_batch(wg, seed=5)
    gs = runtime.GlanceStep(g.weight.to(DEV), g.B, g.L, g.T, DEV, context_p=0.5)
    prev = torch.where(torch.arange(g.L)[None, :] < g.output_length[:, None], 3, 1)
    gs.load(g.hidden.pin_memory(), g.links.pin_memory(), g.output_length.pin_memory(), g.targets.pin_memory(),
            g.target_length.pin_memory(), prev.pin_memory())
    for _ in range(2):
        tree, ll, am, glance = gs.run()
        tree, ll, am = tree.clone(), ll.clone(), am.clone()
    noise = gs.noise.cpu()
    assert noise.std() > 0.5  # drawn inside the replayed graph
    want = pyref.glance_select(tree.cpu(), am.cpu(), g.targets, prev, g.target_length, noise, 0.5)
    for key, val in want.items():
        assert torch.equal(glance[key].cpu(), val), key
    em = ops.proj_logsoftmax_gather(g.hidden.to(DEV), g.weight.to(DEV), g.targets.to(DEV), g.output_length.to(DEV),
                                    g.target_length.to(DEV), want_max=True)
    tree2, ll2 = ops.cuda_pcfg_best_tree(em["match"], g.links.to(DEV), g.output_length.to(DEV), g.target_length.to(DEV))
    assert torch.equal(tree, tree2) and torch.equal(ll, ll2) and torch.equal(am, em["argmax"])
    So, Co = oracle.pcfg_loss(em["match"].cpu().numpy(), g.links.numpy(), g.output_length.numpy(), g.target_length.numpy())
    want_tree = oracle.pcfg_best_tree(So, Co, em["match"].cpu().numpy(), g.links.numpy(), g.output_length.numpy(),
                                      g.target_length.numpy())
    # same emissions; the tables differ from the oracle's only in the last ulp of expf/logf
    assert (tree.cpu().numpy() == want_tree).mean() > 0.99


# ---- criterion glue against the reference criterion's own code (tests/golden/host_criterion.npz) -----------------

@pytest.mark.parametrize("tag,strategy", [("none", None), ("number_random", "number-random"), ("cmlm", "cmlm")])
def test_glance_select_against_reference_criterion(ops, tag, strategy):
    g = _g("host_criterion.npz")
    t = lambda key: torch.from_numpy(g[key]).to(DEV)
    B, L = g["path"].shape
    noise, uniform = pyref.criterion_draws(strategy, int(g[f"{tag}_seed"]), B, L)
    k = ops.get_pcfg_kernel()
    pred = t("logits").argmax(-1)
    got = k.glance_select(t("path"), pred, t("tgt"), t("prev"), t("tgt_len"),
                          None if noise is None else noise.to(DEV), 0.5, strategy,
                          None if uniform is None else uniform.to(DEV))
    assert torch.equal(got["matchmask"], t(f"{tag}_matchmask"))
    assert torch.equal(got["keep_word_mask"], t(f"{tag}_keep"))
    assert torch.equal(got["glat_prev_output_tokens"], t(f"{tag}_glat_prev"))
    accu = float(got["same_num"].sum() / t("tgt_len").sum())
    assert abs(accu - float(g[f"{tag}_glat_accu"])) < 1e-6
    want = pyref.glance_select(t("path").cpu(), pred.cpu(), t("tgt").cpu(), t("prev").cpu(), t("tgt_len").cpu(), noise,
                               0.5, strategy, uniform)
    for key, val in want.items():
        assert torch.equal(got[key].cpu(), val), key


def test_force_emit_against_reference_criterion(pkg, ops, syn):
    g = _g("host_criterion.npz")
    t = lambda key: torch.from_numpy(g[key]).to(DEV)
    eos = syn.eos_mask_(t("match_plain").clone(), t("out_len"), t("tgt_len"))
    assert torch.equal(eos, t("plain_loss_match"))
    ma = eos.clone().requires_grad_(True)
    out = ops.force_emit_mask(ma, t("number_random_matchmask"), t("number_random_keep"))
    assert torch.equal(out.detach(), t("force_loss_match"))
    # the same recording loss as the fixture's: linear with weights loss_w on the finite entries
    n = t("tgt_len").float()
    fin = torch.isfinite(out)
    sent = (torch.where(fin, out, torch.zeros_like(out)) * t("loss_w")).sum((1, 2))
    valid = torch.tensor([True, True, False, True, True], device=DEV)
    (-(torch.where(valid, sent, torch.zeros_like(sent)) / n).mean()).backward()
    torch.testing.assert_close(ma.grad, t("force_match_grad"), rtol=1e-6, atol=0)
    # in place, as the step object uses it
    k = ops.get_pcfg_kernel()
    buf = eos.clone()
    k.force_emit(buf, t("number_random_matchmask"), t("number_random_keep"), out=buf)
    assert torch.equal(buf, t("force_loss_match"))


def test_loss_step_with_force_emit_matches_operator_chain(pkg, ops, syn):
    """GlanceStep -> LossStep(force_emit=True), as a GLAT training step chains them, against the operators one by
    one with autograd and against the oracle fed the masked emissions."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("fe", batch=5, vocab=2000, hidden=64, src_min=6, src_max=20, kind="glance")
    b = syn.make_batch(w, seed=6)
    weight = b.weight.to(DEV)
    prev = torch.where(torch.arange(b.L)[None, :] < b.output_length[:, None], 3, 1)
    gs = runtime.GlanceStep(weight, b.B, b.L, b.T, DEV, context_p=0.5)
    gs.load(b.hidden, b.links, b.output_length, b.targets, b.target_length, prev)
    tree, ll, am, glance = gs.run()
    assert glance["keep_word_mask"].any()
    ls = runtime.LossStep(weight, b.B, b.L, b.T, DEV, force_emit=True)
    ls.load(b.hidden, b.links, b.output_length, b.targets, b.target_length, glance["matchmask"], glance["keep_word_mask"])
    for _ in range(2):  # capture, replay
        stats, mg, lg, loss = [x.clone() for x in ls.run()]
    em = ops.proj_logsoftmax_gather(b.hidden.to(DEV), weight, b.targets.to(DEV), b.output_length.to(DEV),
                                    b.target_length.to(DEV))["match"].requires_grad_(True)
    lk = b.links.to(DEV).requires_grad_(True)
    masked = ops.force_emit_mask(em, glance["matchmask"], glance["keep_word_mask"])
    loss2 = ops.cuda_pcfg_loss(masked, lk, b.output_length.to(DEV), b.target_length.to(DEV))
    loss2.sum().backward()
    assert torch.isfinite(loss2).all()
    assert torch.equal(loss, loss2.detach()) and torch.equal(mg, em.grad) and torch.equal(lg, lk.grad)
    assert (mg[glance["keep_word_mask"]] == 0).all()
    m_np = masked.detach().cpu().numpy()
    So, Co = oracle.pcfg_loss(m_np, b.links.numpy(), b.output_length.numpy(), b.target_length.numpy())
    np.testing.assert_allclose(loss.cpu().numpy(), So[:, 0, 0], rtol=1e-4)
    mgo, lgo = oracle.pcfg_loss_backward(np.ones(b.B, np.float32), So, Co, m_np, b.links.numpy(),
                                         b.output_length.numpy(), b.target_length.numpy())
    mgo[glance["keep_word_mask"].cpu().numpy()] = 0
    np.testing.assert_allclose(mg.cpu().numpy(), mgo, rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy(), lgo, rtol=1e-3, atol=2e-6)


# ---- linear-space loss forward + backward (the default of the fused entry point) ---------------------------------

def _fused(ops, ma, lk, ol, tl):
    k = ops.get_pcfg_kernel()
    loss, mg, lg = k.pcfg_loss_fwd_bwd(ma, lk, ol, tl)
    torch.cuda.synchronize()
    return loss, mg, lg


@pytest.mark.parametrize("peak", [1.0, 8.0, 25.0])
@pytest.mark.parametrize("shape", [dict(batch=5, src_min=4, src_max=30), dict(batch=3, fixed_graph=384, fixed_target=90),
                                   dict(batch=70, src_min=6, src_max=20)])
def test_linear_space_loss_against_oracle_peaked_inputs(ops, syn, monkeypatch, peak, shape):
    """Emissions and transitions sharpened by `peak` (a trained model is far from the near-uniform synthetic
    inputs): columns then span many e-folds, which is what the per-column scaling has to absorb; whatever it
    cannot is recomputed in log space.  Either way the results hold the parity tolerances."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    w = syn.Workload("lin", vocab=50, hidden=8, emissions="logits", **shape)
    b = syn.make_batch(w, seed=31)
    b.logits.mul_(peak)
    ma = syn.reference_match_all(b)
    lk = torch.log_softmax((b.links * peak).view(b.B, b.L, -1), -1).view_as(b.links)
    lk = torch.where(torch.isfinite(b.links), lk, b.links).contiguous()
    lk = torch.where(torch.isnan(lk), torch.full_like(lk, float("-inf")), lk)
    ol, tl = b.output_length.numpy(), b.target_length.numpy()
    So, Co = oracle.pcfg_loss(ma.numpy(), lk.numpy(), ol, tl)
    mgo, lgo = oracle.pcfg_loss_backward(np.ones(b.B, np.float32), So, Co, ma.numpy(), lk.numpy(), ol, tl)
    ops.read_status(DEV)
    loss, mg, lg = _fused(ops, ma.to(DEV), lk.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV))
    recomputed = bool(ops.read_status(DEV) & 16)  # PCFGNAT_STATUS_RECOMPUTED
    assert peak > 1.0 or not recomputed  # ordinary inputs stay in linear space
    assert np.isfinite(So[:, 0, 0]).all()
    np.testing.assert_allclose(loss.cpu().numpy(), So[:, 0, 0], rtol=1e-4)
    np.testing.assert_allclose(mg.cpu().numpy(), mgo, rtol=1e-3, atol=2e-6)
    np.testing.assert_allclose(lg.cpu().numpy(), lgo, rtol=1e-3, atol=2e-6)
    # and against the log-space kernels of the same library
    monkeypatch.setenv("PCFGNAT_LINEAR_DP", "0")
    loss2, mg2, lg2 = _fused(ops, ma.to(DEV), lk.to(DEV), b.output_length.to(DEV), b.target_length.to(DEV))
    torch.testing.assert_close(loss, loss2, rtol=1e-5, atol=0)
    torch.testing.assert_close(mg, mg2, rtol=1e-3, atol=2e-6)
    torch.testing.assert_close(lg, lg2, rtol=1e-3, atol=2e-6)


def test_linear_space_loss_hands_unusual_sentences_to_the_log_space_kernels(ops, syn, monkeypatch):
    """One batch with everything the linear-space kernels do not take themselves: an emission far beyond the range of
    exp() relative to its token's maximum, an out-of-range length, an odd graph length, a single target token, an infeasible sentence (more tokens
    than the graph can emit), next to ordinary sentences.  Every sentence must come out as the log-space kernels
    alone give it, and output buffers that were dirty must be fully overwritten."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    w = syn.Workload("lin2", batch=8, vocab=50, hidden=8, src_min=5, src_max=12, emissions="logits")
    b = syn.make_batch(w, seed=32)
    ma = syn.reference_match_all(b)
    ol, tl = b.output_length.clone(), b.target_length.clone()
    ma[0, 2, 0] = 200.0           # a leaf emission far above the main chain's: exp() overflows
    ol[1] = b.L + 4               # out of range
    ol[2] = ol[2] - 1             # odd graph length
    tl[3] = 1                     # one target token
    tl[4] = min(int(ol[4]) - 1, b.T)  # infeasible: n > m - 2
    k = ops.get_pcfg_kernel()
    args = (ma.to(DEV), b.links.to(DEV), ol.to(DEV), tl.to(DEV))
    ops.read_status(DEV)
    loss, mg, lg = _fused(ops, *args)
    st = ops.read_status(DEV)
    assert st & 1 and st & 16  # a bad length was seen; sentences were recomputed in log space
    monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")  # the kernels that pick up the marked sentences, on their own
    loss2, mg2, lg2 = _fused(ops, *args)
    ops.read_status(DEV)
    assert torch.equal(torch.isfinite(loss), torch.isfinite(loss2))
    fin = torch.isfinite(loss2)
    assert fin[5:].all() and not fin[1] and not fin[4]
    torch.testing.assert_close(loss[fin], loss2[fin], rtol=1e-5, atol=0)
    torch.testing.assert_close(mg, mg2, rtol=1e-3, atol=2e-6, equal_nan=True)
    torch.testing.assert_close(lg, lg2, rtol=1e-3, atol=2e-6, equal_nan=True)
    for i in (0, 1, 2, 3, 4):  # handed over: bit for bit what the log-space kernels give
        assert torch.equal(mg[i].nan_to_num(7.0), mg2[i].nan_to_num(7.0)) and torch.equal(lg[i].nan_to_num(7.0), lg2[i].nan_to_num(7.0))


@pytest.mark.parametrize("B, odd", [(1, 0), (6, 6), (90, 0), (90, 89), (160, 40)])
def test_outside_pass_that_starts_before_the_inside_pass_has_ended(ops, syn, monkeypatch, B, odd):
    """The outside pass stages its inputs while the inside pass is at work, and its clusters without work (odd graph lengths
    here, or fewer sentences than clusters) leave early: repeated calls over the same buffers, and a captured one, give bit for
    bit what a call alone gives, and the sentences handed over are those of the log-space kernels."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_LINEAR_DP", raising=False)
    b = syn.make_batch(syn.Workload("early", batch=B, vocab=50, hidden=8, src_min=4, src_max=24, emissions="logits"), seed=41)
    ma, lk, tl = syn.reference_match_all(b).to(DEV), b.links.to(DEV), b.target_length.to(DEV)
    ol = b.output_length.to(DEV)
    ol[:odd] -= 1
    ops.read_status(DEV)
    want = [x.clone() for x in _fused(ops, ma, lk, ol, tl)]
    assert bool(ops.read_status(DEV) & 16) == (odd > 0)  # PCFGNAT_STATUS_RECOMPUTED
    k = ops.get_pcfg_kernel()
    got = [k.pcfg_loss_fwd_bwd(ma, lk, ol, tl) for _ in range(4)]  # no synchronisation in between
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got.append(k.pcfg_loss_fwd_bwd(ma, lk, ol, tl))
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    for out in got:
        for x, y in zip(out, want):
            assert torch.equal(x.nan_to_num(7.0), y.nan_to_num(7.0))
    if odd:
        monkeypatch.setenv("PCFGNAT_DP_KERNEL", "rows")
        for x, y in zip(_fused(ops, ma, lk, ol, tl), want):
            assert torch.equal(x[:odd].nan_to_num(7.0), y[:odd].nan_to_num(7.0))
    ops.read_status(DEV)


@pytest.mark.parametrize("B", [2, 90])
def test_early_outside_pass_behind_a_kernel_that_makes_the_emissions(B):
    """With every kernel of the chain launched early (PCFGNAT_PDL=1, read once per process): the outside pass stages emissions that
    the projection's last kernel has just written.  Batches follow one another without a synchronisation, each with other emissions
    in the same memory; losses and gradients bit for bit those of calls that wait for one another."""
    import subprocess
    import sys

    from conftest import ROOT

    program = f"""
import torch, __graft_entry__ as entry
syn = entry.load_package().synthetic
from pcfg_nat_b200.custom_ops import pcfg_loss as ops
b = syn.make_batch(syn.Workload("chain", batch={B}, vocab=1000, hidden=64, src_min=6, src_max=30, hidden_std=1.0), seed=5)
d = lambda t: t.to("cuda:0")
hidden, weight, links, ol, targets, tl = map(d, (b.hidden, b.weight, b.links, b.output_length, b.targets, b.target_length))
k = ops.get_pcfg_kernel()
states = [torch.roll(hidden, i, 0) * (1 + i / 8) for i in range(6)]
def batch(h, wait):
    match = k.proj_logsoftmax_gather(h, weight, targets, ol, tl)["match"]
    if wait: torch.cuda.synchronize()
    return k.pcfg_loss_fwd_bwd(match, links, ol, tl)
want = [[x.clone() for x in batch(h, True)] for h in states]
torch.cuda.synchronize()
got = [batch(h, False) for _ in range(3) for h in states]
torch.cuda.synchronize()
for i, out in enumerate(got):
    assert all(torch.equal(x.nan_to_num(7.0), y.nan_to_num(7.0)) for x, y in zip(out, want[i % 6])), i
"""
    env = dict(os.environ, PCFGNAT_PDL="1")
    r = subprocess.run([sys.executable, "-c", program], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("B, L, T", [(20, 314, 238), (1, 322, 304), (2, 384, 238)])
def test_linear_space_loss_at_the_limit_of_shared_memory(ops, monkeypatch, B, L, T):
    """Shapes whose tables come within a hundred bytes of the shared memory that the kernels' own variables leave."""
    monkeypatch.delenv("PCFGNAT_DP_KERNEL", raising=False)
    monkeypatch.delenv("PCFGNAT_LINEAR_DP", raising=False)
    g = torch.Generator(DEV).manual_seed(L)
    match = torch.randn(B, L, T, device=DEV, generator=g) - 6
    links = torch.randn(B, L, 2, L, device=DEV, generator=g)
    at = torch.arange(L, device=DEV)
    allowed = (at[:, None] % 2 == 1) & (at[None, :] % 2 == 1) & (at[None, :] > at[:, None])
    links.masked_fill_(~allowed[None, :, None, :], float("-inf"))
    links = torch.log_softmax(links.flatten(2), -1).nan_to_num(nan=float("-inf"), neginf=float("-inf")).view_as(links)
    ol, tl = torch.full((B,), L, device=DEV), torch.full((B,), T, device=DEV)
    ops.read_status(DEV)
    got = _fused(ops, match, links, ol, tl)
    assert ops.read_status(DEV) & ~16 == 0  # PCFGNAT_STATUS_RECOMPUTED
    monkeypatch.setenv("PCFGNAT_LINEAR_DP", "0")
    want = _fused(ops, match, links, ol, tl)
    torch.testing.assert_close(got[0], want[0], rtol=1e-5, atol=0)
    for x, y in zip(got[1:], want[1:]):
        torch.testing.assert_close(x, y, rtol=1e-3, atol=2e-6)


def test_pipelined_steps_overlap_copies_without_mixing_batches(pkg, ops, syn):
    """Two step objects in turn (copies of the next batch while the current one is computed): different batches
    through the pipeline come out exactly as through a single step object, in order."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("pipe", batch=6, vocab=3000, hidden=128, fixed_graph=40, fixed_target=9, hidden_std=1.0)
    batches = [syn.make_batch(w, seed=40 + i) for i in range(5)]
    weight = batches[0].weight.to(DEV)
    B, L, T = batches[0].B, batches[0].L, batches[0].T
    host = [[t.contiguous().pin_memory() for t in (b.hidden, b.links, b.output_length, b.targets, b.target_length)]
            for b in batches]
    single = runtime.LossStep(weight, B, L, T, DEV)
    want = []
    for h in host:
        single.load(*h)
        want.append([t.clone() for t in single.run()])
    pipe = runtime.PipelinedStep(lambda: runtime.LossStep(weight, B, L, T, DEV))
    got = []
    for h in host:
        pipe.load(*h)
        out = pipe.run()
        got.append([t.clone() for t in out])  # cloned on the run's stream, before the run after next reuses the buffers
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            assert torch.equal(x, y)
    assert not torch.equal(want[0][3], want[1][3])


# ---- lookahead / greedy decoding ---------------------------------------------------------------------------------

@pytest.mark.parametrize("name", ["look_b1_a", "look_b1_b", "greedy_b4", "greedy_b1"])
def test_lookahead_decode_against_reference_model(ops, name):
    g = _g("host_lookahead.npz")
    t = lambda key: torch.from_numpy(g[f"{name}_{key}"]).to(DEV)
    strategy = "lookahead" if int(g[f"{name}_lookahead"]) else "greedy"
    k = ops.get_pcfg_kernel()
    ops.read_status(DEV)
    out, cnt = k.lookahead_decode_device(t("links"), t("ob"), t("tok"), t("out_len"), t("mask"), 1,
                                         float(g[f"{name}_beta"]), strategy)
    want = g[f"{name}_result"]
    assert int(cnt.max()) == want.shape[1]
    assert np.array_equal(out[:, :want.shape[1]].cpu().numpy(), want)
    assert (out[:, want.shape[1]:] == 1).all() and ops.read_status(DEV) == 0


@pytest.mark.parametrize("strategy", ["lookahead", "greedy"])
def test_lookahead_decode_step_against_restatement(pkg, ops, syn, strategy):
    """DecodeStep with the two host-loop strategies of the model, on a ragged batch, against the restatement fed the
    kernel's own emissions (arg-max decoding on identical numbers: exact)."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("la", batch=9, vocab=2000, hidden=64, src_min=4, src_max=40, kind="viterbi")
    b = syn.make_batch(w, seed=8)
    weight = b.weight.to(DEV)
    step = runtime.DecodeStep(weight, b.B, b.L, b.left_tree_mask, DEV, strategy=strategy, decode_beta=0.7)
    step.load(b.hidden, b.links, b.output_length)
    for _ in range(2):
        tokens, count = [x.clone() for x in step.run()]
    em = ops.proj_logsoftmax_gather(b.hidden.to(DEV), weight, None, b.output_length.to(DEV), None, want_max=True)
    rows = pyref.lookahead_decode(b.links, em["max_lprob"].cpu(), em["argmax"].cpu(), b.output_length,
                                  b.left_tree_mask.bool(), 1, 0.7, strategy == "lookahead")
    assert min(len(r) for r in rows) >= 2
    for i, r in enumerate(rows):
        assert int(count[i]) == len(r) and tokens[i, :len(r)].cpu().tolist() == r
        assert (tokens[i, len(r):] == 1).all()


@pytest.mark.parametrize("L", [2, 3, 16, 17, 33, 128, 129, 300])
def test_lookahead_decode_cluster_edges(pkg, ops, L):
    """Sentence counts and graph lengths around the nodes a CTA and a cluster take, with ties, a length of zero, an
    emitted pad token and an invalid length (flagged, nothing decoded)."""
    import importlib

    lm = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)[0]
    g = torch.Generator().manual_seed(L)
    B = 5
    links = torch.randint(-6, 0, (B, L, 2, L), generator=g).float() / 2  # ties
    at = torch.arange(L)
    links.masked_fill_(~((at[:, None] % 2 == 1) & (at[None, :] % 2 == 1) & (at[None, :] > at[:, None]))[None, :, None, :],
                       float("-inf"))
    ob = torch.randint(-4, 0, (B, L), generator=g).float()
    tok = torch.randint(1, 9, (B, L), generator=g)
    ol = torch.tensor([L, max(2, L // 2), max(1, L - 1), 0, L])
    links.masked_fill_((at[None, :] >= ol[:, None])[:, None, None, :], float("-inf"))
    k = ops.get_pcfg_kernel()
    ops.read_status(DEV)
    for strategy in ("lookahead", "greedy"):
        out, cnt = k.lookahead_decode_device(links.to(DEV), ob.to(DEV), tok.to(DEV), ol.to(DEV), lm.to(DEV), 1, 0.5, strategy)
        rows = pyref.lookahead_decode(links, ob, tok, ol, lm.bool(), 1, 0.5, strategy == "lookahead")
        for i, r in enumerate(rows):
            assert int(cnt[i]) == len(r) and out[i].cpu().tolist() == r + [1] * (L - len(r))
    assert ops.read_status(DEV) == 0
    ol[4] = L + 1
    out, cnt = k.lookahead_decode_device(links.to(DEV), ob.to(DEV), tok.to(DEV), ol.to(DEV), lm.to(DEV), 1, 0.5, "greedy")
    assert ops.read_status(DEV) != 0 and int(cnt[4]) == 0 and (out[4] == 1).all()


def test_lookahead_decode_longest_graph(ops):
    """The largest graph whose words and stack fit a CTA's shared memory: 29 056 nodes."""
    L = 29056
    links = torch.full((1, L, 2, L), float("-inf"), device=DEV)
    chain = torch.tensor([1, 9, 20001, L - 1], device=DEV)
    links[0, chain[:-1], 0, chain[1:]] = -1.0
    mask = torch.zeros(L, L, dtype=torch.int64, device=DEV)  # every node may descend to node 0, which emits nothing
    tok = torch.arange(L, device=DEV)[None] + 4
    ops.read_status(DEV)
    out, cnt = ops.get_pcfg_kernel().lookahead_decode_device(links, torch.zeros(1, L, device=DEV), tok,
                                                             torch.tensor([L], device=DEV), mask, 1, 1.0, "greedy")
    assert out[0, :int(cnt[0])].tolist() == [5, 13, 20005, L + 3] and ops.read_status(DEV) == 0


def test_a_refused_shape_leaves_no_error_behind(ops):
    """A graph too large for the shared memory is refused, and the next launches find no error of its."""
    L = 29064
    k = ops.get_pcfg_kernel()
    links = torch.zeros(1, L, 2, L, device=DEV)
    tok = torch.zeros(1, L, dtype=torch.int64, device=DEV)
    with pytest.raises(RuntimeError, match="too large"):
        k.lookahead_decode_device(links, None, tok, torch.tensor([L], device=DEV), torch.zeros(8, 8, device=DEV), 1, 1.0, "greedy")
    rows = torch.ones(2, 8, dtype=torch.float16, device=DEV)
    assert (k.rows_to_bf16(rows) == 1).all()


def test_lookahead_decode_near_ties(pkg, ops):
    """Two candidates per node whose scores differ by the last bit or not at all, with a beta that is not a power of two:
    the choice is the one of separately rounded products and sums, not of fused ones."""
    import importlib

    B, L, beta = 64, 34, 0.7
    lm = importlib.import_module("pcfg_nat_b200.support_tree").get_mask(L, 1)[0]
    g = torch.Generator().manual_seed(5)
    ob = torch.randn(B, L, generator=g) * 3 - 6
    links = torch.full((B, L, 2, L), float("-inf"))
    fused_differs = 0
    for a in range(1, L - 4, 2):
        c1, c2 = a + 2, a + 4
        links[:, a, 0, c1] = torch.randn(B, generator=g) - 4
        links[:, a, 0, c2] = (links[:, a, 0, c1] + ob[:, c1] * beta) - ob[:, c2] * beta
        exact = [(links[:, a, 0, c].double() + ob[:, c].double() * torch.tensor(beta).double()).float() for c in (c1, c2)]
        split = [links[:, a, 0, c] + ob[:, c] * beta for c in (c1, c2)]
        fused_differs += int(((exact[1] > exact[0]) != (split[1] > split[0])).sum())
    assert fused_differs > 50
    tok = torch.arange(L).expand(B, L) + 4
    ol = torch.full((B,), L)
    out, cnt = ops.get_pcfg_kernel().lookahead_decode_device(links.to(DEV), ob.to(DEV), tok.to(DEV), ol.to(DEV), lm.to(DEV), 1,
                                                             beta, "lookahead")
    rows = pyref.lookahead_decode(links, ob, tok, ol, lm.bool(), 1, beta)
    for i, r in enumerate(rows):
        assert int(cnt[i]) == len(r) and out[i].cpu().tolist() == r + [1] * (L - len(r))


def test_loss_step_from_link_features_matches_autograd_chain(pkg, ops, syn):
    """LossStep fed with the projected link features (transitions formed and differentiated inside the step) against
    the operators chained by autograd: extract_links -> cuda_pcfg_loss -> backward."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    support = importlib.import_module("pcfg_nat_b200.support_tree")
    w = syn.Workload("lf", batch=5, vocab=2000, hidden=64, src_min=5, src_max=14)
    b = syn.make_batch(w, seed=9)
    heads, dim = 4, 16
    g = torch.Generator().manual_seed(3)
    q, kl, kr = (torch.randn(b.B, b.L, heads, dim, generator=g).half() for _ in range(3))
    gates = torch.randn(b.B, b.L, heads, generator=g)
    prev = torch.where(torch.arange(b.L)[None, :] < b.output_length[:, None], 3, 1)
    lm, rm, mc = support.get_mask(b.L, 1)
    weight = b.weight.to(DEV)
    step = runtime.LossStep(weight, b.B, b.L, b.T, DEV, link_features=(heads, dim), left_tree_mask=lm, right_tree_mask=rm,
                            main_chain=mc)
    step.load(b.hidden, q, kl, kr, gates, prev, b.output_length, b.targets, b.target_length)
    for _ in range(2):  # capture, replay
        stats, mg, (dq, dkl, dkr, dgates), loss = step.run()
    torch.cuda.synchronize()
    leaves = [x.to(DEV).requires_grad_(True) for x in (q, kl, kr)]
    gt = gates.to(DEV).requires_grad_(True)
    links = ops.get_pcfg_kernel().extract_links(*leaves, gt, prev.to(DEV), 1, lm, rm, mc)
    em = ops.proj_logsoftmax_gather(b.hidden.to(DEV), weight, b.targets.to(DEV), b.output_length.to(DEV),
                                    b.target_length.to(DEV))["match"]
    loss2 = ops.cuda_pcfg_loss(em, links, b.output_length.to(DEV), b.target_length.to(DEV))
    assert torch.isfinite(loss2).all()
    loss2.sum().backward()
    assert torch.equal(loss, loss2.detach())
    for got, leaf in zip((dq, dkl, dkr), leaves):
        torch.testing.assert_close(got, leaf.grad.float(), rtol=1e-3, atol=1e-3)  # the chain rounds its gradients to f16
    torch.testing.assert_close(dgates, gt.grad, rtol=1e-5, atol=1e-6)
    assert dq.abs().sum() > 0 and dkr.abs().sum() > 0


def test_steps_from_link_features_live_side_by_side(pkg, ops, syn):
    """A captured step keeps the node lists that its graph reads: building a second step, of another shape, and letting
    the allocator hand out what was freed leaves the first step's results as they were."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    support = importlib.import_module("pcfg_nat_b200.support_tree")
    heads, dim = 2, 8

    def decode_step(src_max, seed):
        b = syn.make_batch(syn.Workload("side", batch=3, vocab=300, hidden=64, src_min=4, src_max=src_max), seed=seed)
        g = torch.Generator().manual_seed(seed)
        feats = [torch.randn(b.B, b.L, heads, dim, generator=g) for _ in range(3)]
        gates = torch.randn(b.B, b.L, heads, generator=g)
        prev = torch.where(torch.arange(b.L)[None, :] < b.output_length[:, None], 3, 1)
        lm, rm, mc = support.get_mask(b.L, 1)
        step = runtime.DecodeStep(b.weight.to(DEV), b.B, b.L, lm, DEV, link_features=(heads, dim), right_tree_mask=rm,
                                  main_chain=mc, strategy="greedy")
        step.load(b.hidden, *feats, gates, prev, b.output_length)
        return step

    def held(step):  # host copies: nothing of the step is kept by accident
        return [t.cpu() for t in step.run()]

    first = decode_step(12, 1)
    want = held(first)
    nodes, slot_of = first.chain
    assert nodes.tolist() == list(range(1, first.L, 2)) and int(slot_of.max()) == first.L // 2 - 1
    second = decode_step(6, 2)
    held(second)
    filler = [torch.zeros(n, dtype=torch.int32, device=DEV) for n in (8, 16, 24, 48) for _ in range(64)]
    assert all(torch.equal(x, y) for x, y in zip(held(first), want)), len(filler)


@pytest.mark.parametrize("mode", ["links", "all"])
def test_overlapped_load_fetching_from_host_buffers(pkg, ops, syn, mode):
    """An overlapped load whose large inputs are fetched by the kernel that reads the pinned host buffers itself
    (only the real nodes' states / only the transitions the tree masks leave finite) gives the step exactly what the
    plain copies give it, batch after batch (shorter sentences after longer ones: nothing stale is read)."""
    import importlib

    runtime = importlib.import_module("pcfg_nat_b200.runtime")
    w = syn.Workload("fh", batch=6, vocab=3000, hidden=128, src_min=3, src_max=12, hidden_std=1.0)
    batches = [syn.make_batch(w, seed=50 + i) for i in range(4)]
    L, T = max(b.L for b in batches), max(b.T for b in batches)

    def padded(b):
        hid = torch.randn(b.B, L, w.hidden).half()  # garbage beyond the real nodes: it must not matter
        hid[:, :b.L] = b.hidden
        lk = torch.full((b.B, L, 2, L), float("-inf"))
        lk[:, :b.L, :, :b.L] = b.links
        tg = torch.ones(b.B, T, dtype=torch.long)
        tg[:, :b.T] = b.targets
        return [t.contiguous().pin_memory() for t in (hid, lk, b.output_length, tg, b.target_length)]

    weight = batches[0].weight.to(DEV)
    plain = runtime.LossStep(weight, w.batch, L, T, DEV)
    fetched = runtime.LossStep(weight, w.batch, L, T, DEV)
    fetched.fetch_from_host = mode
    for b in batches:
        args = padded(b)
        plain.load(*args)
        want = [t.clone() for t in plain.run()]
        fetched.load(*args, overlap=True)
        got = fetched.run()
        torch.cuda.synchronize()
        for x, y in zip(got, want):
            assert torch.equal(x, y)
        assert fetched.input_bytes() < plain.input_bytes()
        kernel_links = fetched.links.cpu()
        assert torch.equal(kernel_links, args[1])  # the model's masks leave nothing finite outside what was fetched


def test_smoke_with_dependent_launches_and_ranges_switched_on():
    """PCFGNAT_PDL=1 (programmatic dependent launch along the kernel chain) and PCFGNAT_NVTX=1 are read once per
    process: a fresh interpreter runs the package's smoke check, which compares a step with the oracle, with both on."""
    import subprocess
    import sys

    from conftest import ROOT

    env = dict(os.environ, PCFGNAT_PDL="1", PCFGNAT_NVTX="1")
    r = subprocess.run([sys.executable, "-c", "import __graft_entry__ as g; g.smoke()"], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "smoke ok" in r.stdout
