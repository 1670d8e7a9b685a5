"""The work that users of ispan_b200 have it do, as cases whose time can be measured.

Every case goes through a public entry point with the inputs and the handle (a Context or a Server) that a
program keeps between calls.  The graphs are the package's seeded generators at the shapes of its benchmark
and tests: R-MAT, a social-network shape (one giant SCC), a web-crawl shape (a giant SCC beside many planted
mid-size ones) and batches of independent graphs (R-MAT-like and DAGs of planted cycles, alternating).

All outputs are vertex ids and counts, so they are equal or wrong: there is no exact().

Kinds of case:
  plain    one graph on the device, Context.run: labels and SCC counts
  host     one graph in host memory, labels back in host memory: both CSRs from ordinary memory, or the
           forward CSR alone from pinned memory (the reverse is built on the device)
  batch    many graphs as one disjoint union on the device, Context.run with vbase
  graphs   many separate device graphs in one call, Context.run_graphs
  served   requests submitted one by one to a Server, all of them waited for
"""
import numpy as np
import torch

from ispan_b200 import Context, Server, gen

# Sizes at scale 1 of the generators' social and web shapes, and the largest part of each that is measured:
# the web graph (37 GB of CSR and 55 GB of context at scale 1) is measured up to a fifth of its size.
SOCIAL_V, SOCIAL_E = 41_652_231, 1_735_000_000
WEB_V, WEB_E = 700_000_000, 3_300_000_000


def listed():
    return [
        # the smallest call: a 1,024-vertex graph, where launches and latency are all there is
        {"name": "rmat10", "kind": "plain", "shape": "rmat", "scale": 10, "ef": 16, "off": 4},
        # the reference's own small workload: R-MAT scale 16, edge factor 16, int32 offsets
        {"name": "rmat16", "kind": "plain", "shape": "rmat", "scale": 16, "ef": 16, "off": 4},
        # an ordinary single graph: a million vertices
        {"name": "rmat20", "kind": "plain", "shape": "rmat", "scale": 20, "ef": 13, "off": 8},
        # a large social network: 41.6 M vertices, 1.47 G edges, one giant SCC (the headline workload)
        {"name": "social", "kind": "plain", "shape": "social", "scale": 1.0, "off": 8},
        # a large graph in host memory: forward CSR alone, pinned
        {"name": "social-host", "kind": "host", "shape": "social", "scale": 0.1, "off": 8, "both": False},
        # the drop-in call of a program that loaded its graph from files: both CSRs, ordinary memory
        {"name": "web-host", "kind": "host", "shape": "web", "scale": 0.005, "off": 4, "both": True},
        # a web crawl, small and large: a third giant, half trivial, the rest mid-size SCCs in a DAG
        {"name": "web-small", "kind": "plain", "shape": "web", "scale": 0.0103, "off": 4},
        {"name": "web", "kind": "plain", "shape": "web", "scale": 0.2, "off": 8},
        # a batch job over many graphs of uneven sizes (1,000 to a million vertices)
        {"name": "batch", "kind": "batch", "nseg": 512, "vmin": 1000, "vmax": 1_000_000, "efmin": 8, "efmax": 32,
         "cycle": 1000},
        # a handful of small graphs at once
        {"name": "batch-small", "kind": "batch", "nseg": 23, "vmin": 100, "vmax": 5000, "efmin": 4, "efmax": 12,
         "cycle": 40},
        # separate graphs of uneven sizes handed over in one call
        {"name": "graphs", "kind": "graphs", "nseg": 97, "vmin": 64, "vmax": 200_000, "efmin": 8, "efmax": 32,
         "cycle": 1000},
        # a burst of requests at a server, as many small as large ones
        {"name": "served", "kind": "served", "nseg": 64, "vmin": 64, "vmax": 300_000, "efmin": 8, "efmax": 32,
         "cycle": 1000, "requests": 193},
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["rmat", "rmat", "social", "host", "web", "web", "batch", "batch", "graphs", "served"])
    off = rng.choice([4, 8])
    if kind == "rmat":
        return {"kind": "plain", "shape": "rmat", "scale": rng.randint(8, 21), "ef": rng.randint(4, 24), "off": off}
    if kind == "social":
        return {"kind": "plain", "shape": "social", "scale": round(_log_uniform(rng, 0.001, 0.9), 5), "off": off}
    if kind == "host":
        return {"kind": "host", "shape": rng.choice(["social", "web"]), "off": off,
                "scale": round(_log_uniform(rng, 0.0005, 0.05), 5), "both": rng.random() < 0.5}
    if kind == "web":
        return {"kind": "plain", "shape": "web", "scale": round(_log_uniform(rng, 0.0005, 0.18), 5), "off": off}
    vmin = int(_log_uniform(rng, 64, 2000))
    vmax = int(_log_uniform(rng, 4 * vmin, 400_000))
    efmin = rng.randint(4, 8)
    c = {"kind": kind, "nseg": int(_log_uniform(rng, 4, 300 if kind == "batch" else 90)), "vmin": vmin, "vmax": vmax,
         "efmin": efmin, "efmax": rng.randint(efmin + 1, 32), "cycle": int(_log_uniform(rng, 8, 1000))}
    if kind == "served":
        c["requests"] = c["nseg"] + rng.randint(0, 150)
    return c


def _offsets(case):
    return "int64" if case["off"] == 8 else "int32"


def _make(case, seed):
    if case["shape"] == "rmat":
        return gen.rmat(case["scale"], case["ef"], seed)
    make = gen.social if case["shape"] == "social" else gen.web
    return make(seed=seed, scale=case["scale"])


def _make_batch(case, seed):
    return gen.batch(nseg=case["nseg"], vmin=case["vmin"], vmax=case["vmax"], ef_min=case["efmin"],
                     ef_max=case["efmax"], max_cycle=case["cycle"], seed=seed)


def _counts(st):
    return {k: st[k] for k in ("scc_count", "giant_size", "fw_size", "residual")}


def _capacity(case, n):
    """Labels that a program with n graphs of these sizes keeps room for: four standard deviations above
    their mean sum (log-uniform sizes), and a 256-byte boundary for each."""
    lo, hi = case["vmin"], case["vmax"]
    m = (hi - lo) / np.log(hi / lo)
    sd = (max(0.0, (hi * hi - lo * lo) / (2 * np.log(hi / lo)) - m * m)) ** 0.5
    return int(min(n * hi, n * m + 4 * sd * n ** 0.5)) + 64 * n


def _label_buffers(case, pool, picks):
    """One label buffer per request, all slices of one tensor (each at a 256-byte boundary); None if its
    room is too small."""
    sizes = [(pool[i][0].numel() - 1 + 63) // 64 * 64 for i in picks]
    at = np.concatenate([[0], np.cumsum(sizes)])
    if at[-1] > _capacity(case, len(picks)):
        return None, None
    whole = torch.zeros(_capacity(case, len(picks)), dtype=torch.int32, device="cuda")
    return whole, [whole[int(at[k]):int(at[k]) + pool[i][0].numel() - 1] for k, i in enumerate(picks)]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("plain", "host"):
        g = _make(case, seed)
        V, E = g.V, g.E
        s = {"kind": kind, "ctx": Context(V, E)}
        if kind == "plain":
            s["csr"] = g.to_torch(_offsets(case))
            s["labels"] = torch.empty(V, dtype=torch.int32, device="cuda")
        elif case["both"]:
            c = g.to_host(np.dtype(_offsets(case)))
            s["csr"] = (c.fw_beg, c.fw_adj, c.bw_beg, c.bw_adj)
            s["labels"] = np.empty(V, np.int32)
        else:
            fb, fa, _, _ = g.to_pinned()
            if case["off"] == 4:
                fb = fb.to(torch.int32).pin_memory()
            s["keep"] = (fb, fa)
            s["csr"] = (fb.numpy(), fa.numpy())
            s["labels"] = torch.empty(V, dtype=torch.int32, pin_memory=True).numpy()
        g.free()
        return s
    for again in range(100):
        g = _make_batch(case, seed + 1_000_003 * again)
        if g.V > _capacity(case, case["nseg"]):
            continue  # larger graphs than the program has room for
        if kind == "batch":
            V, E, vbase = g.V, g.E, g.vbase
            csr = g.to_torch("int64")
            g.free()
            whole = torch.zeros(_capacity(case, case["nseg"]), dtype=torch.int32, device="cuda")
            return {"kind": kind, "csr": csr, "vbase": vbase, "ctx": Context(V, E), "whole": whole}
        pool = [g.extract(i, "int32") for i in range(case["nseg"])]
        V, E = g.V, g.E
        g.free()
        picks = range(len(pool))
        if kind == "served":
            picks = [int(i) for i in np.random.default_rng(seed).integers(0, len(pool), case["requests"])]
        whole, outs = _label_buffers(case, pool, picks)
        if whole is None:
            continue
        s = {"kind": kind, "pool": pool, "picks": picks, "outs": outs, "whole": whole}
        if kind == "graphs":
            s["ctx"] = Context(V, E)
        else:
            s["server"] = Server(hbm_budget_bytes=12 << 30)
        return s
    raise RuntimeError("no batch of these sizes fits its room")


def run(state):
    kind = state["kind"]
    if kind in ("plain", "host"):
        labels, st = state["ctx"].run(*state["csr"], labels_out=state["labels"])
        return {"labels": labels, **_counts(st)}
    if kind == "batch":
        _, st = state["ctx"].run(*state["csr"], vbase=state["vbase"], labels_out=state["whole"])
        return {"labels": state["whole"], **_counts(st)}
    if kind == "graphs":
        _, st = state["ctx"].run_graphs(state["pool"], labels_out=state["outs"])
        return {"labels": state["whole"], **_counts(st)}
    srv = state["server"]
    tickets = [srv.submit(*state["pool"][i], out) for i, out in zip(state["picks"], state["outs"])]
    for t in tickets:
        srv.wait(t)
    return {"labels": state["whole"]}


def _size(case):
    """Vertices and edges of a case, as the generators give them in the mean."""
    if "shape" in case:
        if case["shape"] == "rmat":
            n = 1 << case["scale"]
            return n, 0.9 * n * case["ef"]
        n, e = (SOCIAL_V, 0.847 * SOCIAL_E) if case["shape"] == "social" else (WEB_V, WEB_E)
        return n * case["scale"], e * case["scale"]
    lo, hi = case["vmin"], case["vmax"]
    v = (hi - lo) / np.log(hi / lo)  # the mean of a log-uniform draw
    n = case["requests"] if case["kind"] == "served" else case["nseg"]
    ef = 0.5 * (0.75 * (case["efmin"] + case["efmax"]) / 2 + 3)  # half R-MAT-like, half DAGs of planted cycles
    return float(n * v), float(n * v * ef)


def work(case):
    """Both CSR directions read once (forward-only host input: one) and the labels written once."""
    V, E = _size(case)
    off = case.get("off", 8 if case["kind"] == "batch" else 4)
    return {"bytes": float((2 if case.get("both", True) else 1) * (off * V + 4 * E) + 4 * V), "flops": 0.0}
