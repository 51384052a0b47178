"""Workloads of the Tree-SVD refresh, called as a user's program calls it.

Kinds:
  step    one snapshot of a session (edge batch in, embedding out): graph
          insert, PPR refresh + push, log transform, frPCA of the blocks,
          merges. "scratch" pushes from scratch at every snapshot (the
          reference's Plain method, and its run.sh default).
  factor  blocks_factorize + tree_merge of a session whose blocks are
          materialized: the factor stage of one snapshot.
  merge   tree_merge alone: the h-ary merges of given block factors.
  frpca   frPCA of a caller's CSR matrix (host buffers in and out): tensor
          cores ("mixed"), FP32 SpMM ("fp32", the path of the legacy frPCA
          symbol) or the allocation-free entry point ("noalloc").
  svd     merge_svd: the truncated SVD of one dense matrix (host buffers).
  lp      link-prediction scores of vertex pairs.

Graphs are R-MAT (0.57, 0.19, 0.19, 0.05) without self-loops or duplicates,
edges in random time order, as in the package's workloads. Singular vectors
are defined up to sign and, where singular values nearly coincide, up to a
rotation among themselves, so the answers are what a program computes from
them next: the sources' similarity matrix E E^T of the embedding E, and the
rank-k approximation U diag(S) V^T of a matrix with S beside it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "tree-embedding_gb300"))
import tsvd_gb300 as T  # noqa: E402

DELTAS = 24  # edge batches a session holds; a longer run goes round them again

_SESSION = dict(directed=False, h=2, d=128, q=6, rmax=1e-7, transform=T.TRANSFORM_LOG10_NC,
                scratch=False, hubs=False, delta=0)


def listed():
    def session(name, kind, **kw):
        return dict(_SESSION, name=name, kind=kind, **kw)

    return [
        # a small serving tenant taking a batch of a few hundred edges (the
        # smoke workload's sizes): launches and latency count
        session("step_tenant", "step", n=4000, m=30_000, sources=64, parts=4, d=32, rmax=1e-5,
                transform=T.TRANSFORM_LN_N, delta=300),
        # the N = 1e5 workload, a 1 % batch
        session("step_100k", "step", n=100_000, m=1_000_000, sources=500, parts=16, rmax=1e-6,
                transform=T.TRANSFORM_LN_N, delta=10_000),
        # a directed graph of the Patent-sized workload's degree (5), odd sizes
        session("step_patent", "step", n=300_007, m=1_530_000, directed=True, sources=1001,
                parts=64, delta=15_300),
        # a directed graph of the Wikipedia-sized workload's degree (29) with
        # its hub push schedule, a 1 % batch
        session("step_wiki", "step", n=150_001, m=4_300_000, directed=True, sources=1000,
                parts=32, hubs=True, delta=43_000),
        # the Plain method: every snapshot pushed from scratch
        session("recompute_50k", "step", n=50_021, m=400_000, sources=300, parts=8, d=64,
                scratch=True, delta=2_000),
        # factor stage with every block dirty: 64 blocks of about 1500 x 3100
        session("factor_64", "factor", n=200_000, m=2_000_000, sources=1500, parts=64,
                rmax=1e-6),
        # many small blocks (the degree-sorted batched workloads have 256)
        session("factor_256", "factor", n=131_101, m=1_000_000, sources=700, parts=256,
                rmax=1e-6),
        # the reference's run.sh merge arity 8: merges wider than 256 columns
        session("merge_arity8", "merge", n=30_000, m=300_000, sources=1500, parts=64, h=8,
                rmax=1e-6),
        # one block given as CSR, tensor-core products
        dict(name="frpca_block", kind="frpca", rows=1500, cols=6000, density=0.1, k=128, q=6,
             path="mixed"),
        # a small matrix through the legacy symbol's path, odd pass count
        dict(name="frpca_legacy", kind="frpca", rows=600, cols=3001, density=0.05, k=32, q=3,
             path="fp32"),
        # the tree's merge of two rank-128 factors, called alone
        dict(name="svd_600x256", kind="svd", rows=600, cols=256, d=128),
        # scoring a batch of candidate pairs
        dict(name="lp_scores", kind="lp", n=20_000, m=150_000, sources=200, parts=8, d=64,
             directed=True, pairs=20_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "factor", "merge", "frpca", "frpca", "svd", "lp"])
    if kind == "frpca":
        path = rng.choice(["mixed", "fp32", "noalloc"])
        small = path == "noalloc"
        rows = _log(rng, 100, 500 if small else 1500)
        cols = _log(rng, 400, 2000 if small else 6000)
        k = min(_log(rng, 8, 64 if small else 128), rows // 4)
        return dict(kind="frpca", rows=rows, cols=cols, density=rng.uniform(0.03, 0.1), k=k,
                    q=rng.choice([3, 4, 6, 7]), path=path)
    if kind == "svd":
        rows, d = _log(rng, 300, 3000), rng.choice([16, 32, 50, 64, 128])
        return dict(kind="svd", rows=rows, cols=2 * d, d=d)
    if kind == "lp":
        return dict(kind="lp", n=_log(rng, 5000, 20_000), m=150_000, sources=_log(rng, 64, 200),
                    parts=rng.choice([4, 8]), d=rng.choice([32, 64]), directed=True,
                    pairs=_log(rng, 100, 20_000))
    c = dict(_SESSION, kind=kind)
    n = c["n"] = _log(rng, 4000, 150_000)
    c["m"] = int(n * rng.uniform(5, 12))
    c["sources"] = _log(rng, 150, 1000)
    c["d"] = rng.choice([32, 64, 100, 128])
    c["h"] = rng.choice([2, 2, 4]) if kind != "merge" else rng.choice([2, 4, 8])
    c["parts"] = {2: rng.choice([4, 8, 16, 32]), 4: rng.choice([4, 16]), 8: rng.choice([8, 64])}[c["h"]]
    c["d"] = min(c["d"], c["sources"] // 2)
    c["rmax"] = rng.choice([1e-5, 1e-6])
    c["transform"] = rng.choice([T.TRANSFORM_LN_N, T.TRANSFORM_LOG10_NC])
    if kind == "step":
        c["directed"] = rng.random() < 0.5
        c["scratch"] = rng.random() < 0.25
        c["delta"] = max(20, int(c["m"] * rng.uniform(0.001, 0.01)))
    return c


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rmat(n, count, directed, g):
    """`count` distinct edges in random order, (count, 2) int32 on the GPU."""
    levels = max(1, (n - 1).bit_length())
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while keys.numel() < count:
        want = int(1.5 * (count - keys.numel())) + 4096
        a = torch.zeros(want, dtype=torch.int64, device="cuda")
        b = torch.zeros_like(a)
        for _ in range(levels):
            u = torch.rand(want, generator=g, device="cuda")
            a = 2 * a + (u >= 0.76)
            b = 2 * b + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
        if not directed:
            a, b = torch.minimum(a, b), torch.maximum(a, b)
        ok = (a < n) & (b < n) & (a != b)
        keys = torch.unique(torch.cat([keys, a[ok] * n + b[ok]]))
    keys = keys[torch.randperm(keys.numel(), generator=g, device="cuda")[:count]]
    return torch.stack([keys // n, keys % n], 1).to(torch.int32).contiguous()


def _open_session(case, seed, first, g, **kw):
    """A session with its first snapshot done."""
    deg = torch.bincount(first[:, 0].long(), minlength=case["n"])
    if not case["directed"]:
        deg += torch.bincount(first[:, 1].long(), minlength=case["n"])
    live = torch.nonzero(deg > 0).flatten()
    pick = live[torch.randperm(live.numel(), generator=g, device="cuda")[:case["sources"]]]
    s = T.Session(case["n"], pick.to(torch.int32).cpu().numpy(), directed=case["directed"],
                  alpha=0.2, n_parts=case["parts"], rank_d=case["d"], seed=int(seed),
                  dirty_rule=T.DIRTY_ALL, **kw)
    torch.cuda.synchronize()
    s.step_device(first.data_ptr(), first.shape[0])
    return s


def _matrix(rows, cols, density, g):
    """A block-like matrix: positive log-scale entries with row and column
    levels, a decaying low-rank part and noise, zero below a threshold."""
    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    r = 160
    decay = torch.arange(1, r + 1, device="cuda", dtype=torch.float64) ** -0.8
    x = normal(rows, 1) * 0.7 + normal(1, cols) + (normal(rows, r) * decay) @ normal(r, cols)
    x += 0.1 * normal(rows, cols)
    t = torch.sort(x.flatten()[:: max(1, x.numel() // 100_000)])[0]
    x = (x - t[int((1 - density) * (t.numel() - 1))]).clamp_(min=0)
    return x.float().double()


def _merge_matrix(case, g):
    """Two sibling factors U diag(s) with power-law singular values whose
    column spaces overlap, as neighbouring blocks' do."""
    def basis(x):
        return torch.linalg.qr(x)[0]

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    d = case["cols"] // 2
    s = 100 * torch.arange(1, d + 1, device="cuda", dtype=torch.float64) ** -0.7
    shared = normal(case["rows"], d)
    return torch.cat([basis(shared + normal(case["rows"], d)) * s for _ in range(2)], 1).cpu().numpy()


def _session_kw(case):
    kw = dict(rmax=case["rmax"], hierarchy_n=case["h"], passes_q=case["q"],
              transform=case["transform"], lazy_update_start_iter=2,
              dynamic_ppr_start_iter=1 << 30 if case["scratch"] else 2)
    if case["hubs"]:
        kw.update(push_levels=3, push_ratio=4.0, push_hub_degree=1024)
    return kw


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "frpca":
        x = _matrix(case["rows"], case["cols"], case["density"], g)
        at = torch.nonzero(x)
        indptr = torch.zeros(case["rows"] + 1, dtype=torch.int64, device="cuda")
        indptr[1:] = torch.cumsum((x != 0).sum(1), 0)
        return dict(kind=kind, csr=(indptr.cpu().numpy(), at[:, 1].to(torch.int32).cpu().numpy(),
                                    x[at[:, 0], at[:, 1]].cpu().numpy()),
                    shape=(case["rows"], case["cols"]), k=case["k"], q=case["q"],
                    path=case["path"], seed=int(seed))
    if kind == "svd":
        return dict(kind=kind, m=_merge_matrix(case, g), d=case["d"])
    if kind == "lp":
        first = _rmat(case["n"], case["m"], True, g)
        s = _open_session(case, seed, first, g, rmax=1e-6, transform=T.TRANSFORM_LOG10_LP,
                          root_scaling=T.ROOT_U, lp_right_factor=True, lazy_update_start_iter=2)
        rng = np.random.RandomState(int(seed) & 0x7FFFFFFF)
        pairs = np.stack([rng.choice(s.sources, case["pairs"]),
                          rng.randint(0, case["n"], case["pairs"])], 1).astype(np.int32)
        return dict(kind=kind, s=s, pairs=pairs)
    delta = case["delta"]
    edges = _rmat(case["n"], case["m"] + DELTAS * delta, case["directed"], g)
    s = _open_session(case, seed, edges[:case["m"]].contiguous(), g, **_session_kw(case))
    deltas = [edges[case["m"] + i * delta:case["m"] + (i + 1) * delta].contiguous()
              for i in range(DELTAS if delta else 0)]
    return dict(kind=kind, s=s, deltas=deltas, at=0)


class _Factor:
    """The session's device-resident embedding (|S| x d float32)."""

    def __init__(self, s):
        self.__cuda_array_interface__ = dict(shape=(s.S, s.d), typestr="<f4", version=3,
                                             strides=None, data=(s.embedding_device_ptr(), False))


def _similarity(s):
    """E E^T on torch's stream, in order with the session's own."""
    cur, own = torch.cuda.current_stream(), torch.cuda.ExternalStream(s.stream())
    cur.wait_stream(own)
    e = torch.as_tensor(_Factor(s), device="cuda")
    out = e @ e.T
    own.wait_stream(cur)
    return out


def run(state):
    kind = state["kind"]
    if kind == "frpca":
        u, sig, v = T.frpca(*state["csr"], state["shape"], state["k"], state["q"],
                            seed=state["seed"], noalloc=state["path"] == "noalloc",
                            fp32=state["path"] == "fp32")
        # the library's factors are float32 values in the binding's float64 arrays
        f = [torch.from_numpy(x).cuda().float() for x in (u * sig, sig, v)]
        return dict(low_rank=f[0] @ f[2].T, sigma=f[1])
    if kind == "svd":
        us, sig = T.merge_svd(state["m"], state["d"])
        us, sig = (torch.from_numpy(x).cuda().float() for x in (us, sig))
        return dict(gram=us @ us.T, sigma=sig)
    s = state["s"]
    if kind == "lp":
        return s.lp_scores(state["pairs"])
    if kind == "step":
        e = state["deltas"][state["at"]]
        state["at"] = (state["at"] + 1) % len(state["deltas"])
        s.step_device(e.data_ptr(), e.shape[0])
    else:
        if kind == "factor":
            s.blocks_factorize(1)
        s.tree_merge()
    return _similarity(s)


def work(case):
    kind = case["kind"]
    if kind == "frpca":
        m, n, k, q = case["rows"], case["cols"], case["k"], case["q"]
        nnz, l = case["density"] * m * n, case["k"] + 5
        return dict(bytes=12 * nnz + 8 * (m + 1) + 8 * k * (m + n + 1),
                    flops=2 * nnz * l * q + q * (m + n) * l * l)
    if kind == "svd":
        m, n, d = case["rows"], case["cols"], case["d"]
        return dict(bytes=8 * (m * n + m * d + d), flops=2 * m * n * n + 4 * n ** 3 + 2 * m * n * d)
    if kind == "lp":
        return dict(bytes=case["pairs"] * (8 + 8 + 4 * case["d"]) + 4 * case["sources"] * case["d"],
                    flops=2 * case["pairs"] * case["d"])
    n, S, d, h, P = case["n"], case["sources"], case["d"], case["h"], case["parts"]
    l, dirs = d + 5, 2 if case["directed"] else 1
    nodes = (P - 1) // (h - 1)
    b = 4 * S * d * (nodes + P) + 4 * S * S
    f = nodes * (2 * S * (h * d) ** 2 + 2 * S * h * d * d) + 2 * S * S * d
    if kind in ("factor", "step"):
        b += 2 * n * S
        f += 2 * n * S * l * case["q"] + (P * S + n) * l * l * case["q"]
    if kind == "step":
        b += 4 * n * S * dirs + 8 * case["delta"] + 4 * dirs * case["m"]
    return dict(bytes=b, flops=f)


def exact(case, seed):
    g = _generator(seed)
    if case["kind"] == "frpca":
        a = _matrix(case["rows"], case["cols"], case["density"], g).cpu().numpy()
        lam = np.linalg.eigvalsh(a @ a.T if a.shape[0] <= a.shape[1] else a.T @ a)[::-1]
        # the low-rank product of a randomized method is its own, not the
        # truncated SVD's, where singular values decay slowly
        return dict(low_rank=None, sigma=np.sqrt(np.maximum(lam[:case["k"]], 0)))
    if case["kind"] == "svd":
        u, sig, _ = np.linalg.svd(_merge_matrix(case, g), full_matrices=False)
        us = u[:, :case["d"]] * sig[:case["d"]]
        return dict(gram=us @ us.T, sigma=sig[:case["d"]])
    # a push may end in any state whose residues are below rmax, so a
    # snapshot's result has no one exact value
    return None
