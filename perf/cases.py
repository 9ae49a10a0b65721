"""Timed cases of the track finder: what a program that uses it has it do.

Each case is one pass through the public entry points (tracking-itsu_b200/itsu/capi.py over the C
ABI of include/itsu.h), at sizes of the benchmark's configurations and of the tests: a pp-like
collision is 60 tracks, a mid-size one 400, a central Pb-Pb-like one 6000 tracks with 5% noise, the
uneven batch is log-uniform over 20..8000 tracks, a pile-up frame is 5 collisions of about 1500
tracks with 10% noise over shared clusters. Inputs come from the repository's seeded generator.

Outputs of the track finder are records (clusters, tracklets, cells, roads) whose every field is bit
identical to the reference's binary32 arithmetic; they are returned as the 32-bit words of the
records, so that they are compared byte for byte, which is stricter than any rounding bound.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tracking-itsu_b200"))

from itsu import capi, gen, prefilter  # noqa: E402

DEVICE = "cuda:0"
SEED_STRIDE = 100_003  # events of one seed: seed * SEED_STRIDE + index


def listed():
    return [
        # online / simulation loop over single small collisions, one call per event: latency bound
        {"name": "vertex_pp", "kind": "vertex", "events": 8, "tracks": 60, "pt_mean": 0.5, "noise": 0.01},
        # the same loop over central collisions, one at a time (interactive analysis, event display)
        {"name": "vertex_central", "kind": "vertex", "events": 2, "tracks": 6000, "pt_mean": 0.6, "noise": 0.05},
        # the reference's own seam: one call per stage, then every intermediate list back on the host
        {"name": "stages_mid", "kind": "stages", "tracks": 400, "pt_mean": 0.6, "noise": 0.05},
        # high-rate pp reconstruction: many tiny events per device-resident batch
        {"name": "batch_pp", "kind": "batch", "form": "plain", "events": 1024, "tracks": 60, "tracks_max": 60, "noise": 0.01},
        # minimum-bias reconstruction: multiplicities spread over more than two decades in one batch
        {"name": "batch_uneven", "kind": "batch", "form": "plain", "events": 256, "tracks": 20, "tracks_max": 8000, "noise": 0.05},
        # the headline batch: 128 central events resident on the device
        {"name": "batch_central", "kind": "batch", "form": "plain", "events": 128, "tracks": 6000, "tracks_max": 6000, "noise": 0.05},
        # the same events from pinned host records to roads on the host, copies overlapping the work
        {"name": "stream_central", "kind": "stream", "events": 128, "tracks": 6000},
        # pile-up frames from the host, every collision of a frame tracked over the frame's clusters
        {"name": "frames_pileup", "kind": "frames", "calls": 2, "frames": 16, "collisions": 5, "tracks": 1500},
        # the learned form: the trained tracklet gate in front of the plain path
        {"name": "gate_central", "kind": "batch", "form": "gate", "events": 64, "tracks": 6000, "tracks_max": 6000, "noise": 0.05},
        # the learned form's other network: the pair prefilter inside the cell stage
        {"name": "pair_central", "kind": "batch", "form": "pair", "events": 32, "tracks": 6000, "tracks_max": 6000, "noise": 0.05},
        # the clustering stage alone, on the caller's device buffers (a process that cannot allocate)
        {"name": "clustering", "kind": "clustering", "tracks": 6000},
        # retraining the pair prefilter: the full-set gradient (forward and backward), then Adam steps
        {"name": "pair_train", "kind": "train", "samples": 262144, "steps": 50, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vertex", "stages", "batch", "batch", "uneven", "gate", "pair", "stream", "frames", "clustering", "train"])
    if kind == "vertex":
        return {"kind": "vertex", "events": rng.randint(1, 4), "tracks": _log_int(rng, 20, 8000), "pt_mean": 0.6,
                "noise": round(rng.uniform(0.0, 0.1), 3)}
    if kind == "stages":
        return {"kind": "stages", "tracks": _log_int(rng, 20, 6000), "pt_mean": 0.6, "noise": round(rng.uniform(0.0, 0.1), 3)}
    if kind == "batch":  # events of one size, at most the headline batch's tracks in all
        tracks = _log_int(rng, 20, 6000)
        return {"kind": "batch", "form": "plain", "events": _log_int(rng, 1, min(1024, 128 * 6000 // tracks)), "tracks": tracks,
                "tracks_max": tracks, "noise": 0.05}
    if kind == "uneven":
        lo = _log_int(rng, 20, 1000)
        hi = _log_int(rng, 2 * lo, 8000)
        squares = (hi * hi - lo * lo) / (2 * math.log(hi / lo))  # the mean of tracks^2, which the tracklets follow
        return {"kind": "batch", "form": "plain", "events": _log_int(rng, 8, int(min(256, 128 * 6000 ** 2 / squares))), "tracks": lo,
                "tracks_max": hi, "noise": round(rng.uniform(0.0, 0.1), 3)}
    if kind in ("gate", "pair"):
        tracks = _log_int(rng, 500, 6000)
        return {"kind": "batch", "form": kind, "events": _log_int(rng, 1, 64), "tracks": tracks, "tracks_max": tracks, "noise": 0.05}
    if kind == "stream":
        return {"kind": "stream", "events": _log_int(rng, 8, 128), "tracks": _log_int(rng, 1000, 6000)}
    if kind == "frames":
        return {"kind": "frames", "calls": rng.randint(1, 3), "frames": rng.randint(1, 16), "collisions": rng.randint(2, 5),
                "tracks": _log_int(rng, 100, 1500)}
    if kind == "clustering":
        return {"kind": "clustering", "tracks": _log_int(rng, 20, 8000)}
    return {"kind": "train", "samples": _log_int(rng, 4096, 262144), "steps": rng.randint(10, 60), "batch": 32 * rng.randint(32, 256)}


# ---- inputs ----


def _events(case, seed, count):
    """`count` events of the case: its track count, or track counts log-uniform between its two."""
    lo, hi = case["tracks"], case.get("tracks_max", case["tracks"])
    mults = [lo] * count if lo == hi else gen.batch_multiplicities(seed, count, lo, hi)
    return [gen.make_event(seed * SEED_STRIDE + i, int(n), pt_mean=case.get("pt_mean", 0.6), noise=case.get("noise", 0.05))
            for i, n in enumerate(mults)]


def _pinned(array):
    return torch.from_numpy(np.ascontiguousarray(array).reshape(-1).view(np.uint8)).pin_memory()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _road_capacity(tracks):
    """Roads a caller leaves room for per run: the generator's events have about 1.2 per track, small ones up to 3."""
    return 2 * tracks + 512


def _cluster_capacity(tracks):
    """Clusters a caller leaves room for per event: at most 7 per track and the noise, none dropped."""
    return 9 * tracks + 256


def prepare(case, seed):
    kind = case["kind"]
    if kind == "vertex":
        return dict(kind=kind, ctx=capi.Context(), events=_events(case, seed, case["events"]),
                    roads=np.zeros((case["events"], 8 * _road_capacity(case["tracks"])), np.int32))
    if kind == "stages":
        n = case["tracks"]
        clusters, tracklets, cells = _cluster_capacity(n), 10 * n + n * n // 40 + 1024, 15 * n + 2048
        words = dict(clusters=9 * clusters, index_tables=6 * 401, tracklets=4 * tracklets, trk_lookup=clusters, cells=10 * cells,
                     cell_lookup=tracklets, nb_offsets=cells + 4, nb=cells, roads=8 * _road_capacity(n))
        return dict(kind=kind, ctx=capi.Context(), event=_events(case, seed, 1)[0],
                    lists={k: np.zeros(v, np.int32) for k, v in words.items()})
    if kind == "batch":
        ctx = capi.Context()
        events = _events(case, seed, case["events"])
        batch = prefilter.DeviceBatch(ctx, events, torch.device(DEVICE))
        if case["form"] == "gate":
            ctx.gate_set_model(capi.gate_load(prefilter.GATE_CHECKPOINTS["pbpb"]))
            ctx.gate_enable(True)
        elif case["form"] == "pair":
            ctx.prefilter_set_model(capi.prefilter_load(prefilter.CHECKPOINTS["pbpb"]))
            ctx.prefilter_enable(True)
        # room for the largest mean multiplicity of such a batch, whatever this one drew
        room = len(events) * _road_capacity(case["tracks_max"])
        s = dict(kind=kind, ctx=ctx, batch=batch, roads=torch.zeros(8 * room, dtype=torch.int32, device=DEVICE),
                 road_offsets=torch.zeros(len(events) + 1, dtype=torch.int32, device=DEVICE))
        torch.cuda.synchronize()
        return s
    if kind == "stream":
        clusters, offsets, vertices = gen.pack_batch(_events(case, seed, case["events"]))
        n, capacity = case["events"], case["events"] * _road_capacity(case["tracks"])
        return dict(kind=kind, ctx=capi.Context(flags=capi.FLAG_STREAM_HOST), n=n, clusters=_pinned(capi.track_clusters(clusters)),
                    offsets=_pinned(offsets), vertices=_pinned(vertices), capacity=capacity,
                    roads=torch.zeros(capacity * 8, dtype=torch.int32).pin_memory(),
                    road_offsets=torch.zeros(n + 1, dtype=torch.int32).pin_memory())
    if kind == "frames":
        calls = []
        for k in range(case["calls"]):
            frames = gen.pileup_stream(seed * 16 + k + 1, case["frames"], collisions=case["collisions"], n_tracks=case["tracks"])
            packed = gen.pack_frames(frames)
            host = [_pinned(a) for a in packed]
            f = capi.Frames()
            f.clusters, f.frame_offsets, f.vertices, f.vertex_frame = (t.data_ptr() for t in host)
            f.n_frames, f.n_vertices = len(frames), len(packed[3])
            capacity = f.n_vertices * _road_capacity(case["tracks"])
            calls.append(dict(frames=f, host=host, capacity=capacity, roads=torch.zeros(capacity * 8, dtype=torch.int32).pin_memory(),
                              road_offsets=torch.zeros(f.n_vertices + 1, dtype=torch.int32).pin_memory()))
        return dict(kind=kind, ctx=capi.Context(), calls=calls)
    if kind == "clustering":
        ev = gen.make_event(seed * SEED_STRIDE, case["tracks"])
        clusters, offsets, vertex = gen.pack_batch([ev])
        n = len(clusters)
        s = dict(kind=kind, lib=capi.load(), n=n, clusters=torch.from_numpy(clusters.view(np.uint8)).to(DEVICE),
                 offsets=torch.from_numpy(offsets).to(DEVICE), vertex=torch.from_numpy(vertex).to(DEVICE),
                 sorted=torch.zeros((_cluster_capacity(case["tracks"]), 9), dtype=torch.int32, device=DEVICE),
                 tables=torch.zeros((6, 401), dtype=torch.int32, device=DEVICE))
        torch.cuda.synchronize()
        return s
    assert kind == "train"
    model = capi.prefilter_load(prefilter.CHECKPOINTS["pbpb"])
    features, labels = _samples(case, seed, model)
    s = dict(kind=kind, ctx=capi.Context(), model=model, n=case["samples"], features=features.to(DEVICE), labels=labels.to(DEVICE),
             cfg=capi.train_config(steps=case["steps"], batch=case["batch"], seed=seed + 1))
    torch.cuda.synchronize()
    return s


def _samples(case, seed, model):
    """Training samples spread as the model's standardisation says, three quarters of them on roads."""
    rng = torch.Generator().manual_seed(seed)
    mean, scale = torch.tensor(list(model.mean)), 1.0 / torch.tensor(list(model.inv_std))
    x = torch.randn((case["samples"], 8), generator=rng)
    labels = (torch.rand(case["samples"], generator=rng) < torch.sigmoid(1.2 - 1.5 * x[:, 0] - x[:, 5])).to(torch.uint8)
    return (mean + scale * x).contiguous(), labels


# ---- one pass ----


class _DeviceWords:
    """n 32-bit words at a device address, for torch.as_tensor."""

    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (address, False), "version": 2}


def _words(records):
    return np.ascontiguousarray(records).reshape(-1).view(np.int32)


def _keep(buffer, *arrays):
    """The arrays' words one after another at the start of the caller's buffer, zeros after them."""
    n = sum(len(a) for a in arrays)
    np.concatenate(arrays, out=buffer[:n])
    buffer[n:] = 0
    return buffer


def _run_vertex(s):
    return [_keep(s["roads"][k], _words(s["ctx"].clusters_to_tracks(ev.layers, ev.vertices[0]))) for k, ev in enumerate(s["events"])]


def _run_batch(s):
    ctx = s["ctx"]
    ctx.batch_run(s["batch"].batch)
    roads, offsets, n = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_int64()
    ctx._check(ctx.lib.itsu_batch_roads_device(ctx.h, ctypes.byref(roads), ctypes.byref(offsets)))
    ctx._check(ctx.lib.itsu_batch_road_count(ctx.h, ctypes.byref(n)))
    # the roads stay in the context's arena until its next run: copied out for the steps after
    if n.value:
        s["roads"][: 8 * n.value].copy_(torch.as_tensor(_DeviceWords(roads.value, 8 * n.value), device=DEVICE))
    s["road_offsets"].copy_(torch.as_tensor(_DeviceWords(offsets.value, s["batch"].n_runs + 1), device=DEVICE))
    return {"roads": s["roads"], "road_offsets": s["road_offsets"]}


def _run_stages(s):
    r = s["ctx"].run_vertex(s["event"].layers, s["event"].vertices[0])
    lists = {k: [_words(x) for x in (v if isinstance(v, list) else [v])] for k, v in r.items()}
    out = {k: _keep(s["lists"][k], *v) for k, v in lists.items()}
    out["lengths"] = np.array([len(x) for v in lists.values() for x in v], np.int32)
    return out


def _run_stream(s):
    ctx = s["ctx"]
    ctx._check(ctx.lib.itsu_batch_run_host_tracks(ctx.h, _ptr(s["clusters"]), _ptr(s["offsets"]), _ptr(s["vertices"]), s["n"],
                                                  _ptr(s["roads"]), s["capacity"], _ptr(s["road_offsets"])))
    return {"roads": s["roads"], "road_offsets": s["road_offsets"]}


def _run_frames(s):
    ctx = s["ctx"]
    for c in s["calls"]:
        ctx._check(ctx.lib.itsu_frames_run_host(ctx.h, ctypes.byref(c["frames"]), _ptr(c["roads"]), c["capacity"], _ptr(c["road_offsets"])))
    return [{"roads": c["roads"], "road_offsets": c["road_offsets"]} for c in s["calls"]]


def _run_clustering(s):
    st = s["lib"].itsu_pvc_initialize_noalloc(_ptr(s["clusters"]), _ptr(s["offsets"]), _ptr(s["vertex"]), s["n"], _ptr(s["sorted"]),
                                              _ptr(s["tables"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if st != capi.OK:
        raise capi.ItsuError(st, s["lib"].itsu_last_error(None).decode())
    polar = s["sorted"].view(torch.float32)
    return {"sorted": s["sorted"], "tables": s["tables"], "phi": polar[:, 3], "r": polar[:, 4]}


def _run_train(s):
    ctx = s["ctx"]
    ctx.prefilter_set_model(s["model"])
    grad, loss = ctx.prefilter_gradient(s["features"].data_ptr(), s["labels"].data_ptr(), s["n"])
    losses = ctx.prefilter_train(s["features"].data_ptr(), s["labels"].data_ptr(), s["n"], s["cfg"])
    return {"grad": grad, "loss": loss, "losses": losses, "params": ctx.prefilter_get_model().params()}


def run(state):
    kind = state["kind"]
    return {"vertex": _run_vertex, "stages": _run_stages, "batch": _run_batch, "stream": _run_stream, "frames": _run_frames, "clustering": _run_clustering,
            "train": _run_train}[kind](state)


# ---- what a pass cannot do without ----


def _event_work(tracks, clusters, record, keep_lists=True, collisions=1):
    """Bytes and operations of one run over an event: its clusters read once, its lists written once
    (the roads alone where nothing else is kept). List lengths follow the generator's events: 6.5 n +
    0.0086 n^2 tracklets over all n tracks, and 6.5 cells, 5.4 links and 1.2 roads per track of the
    run's own collision."""
    over_all = tracks * collisions
    tracklets, cells, links, roads = 6.5 * over_all + 0.0086 * over_all * over_all, 6.5 * tracks, 5.4 * tracks, 1.2 * tracks
    size = clusters * record + 32 * roads
    if keep_lists:  # sorted clusters, index tables, tracklets and cells with their lookup tables, neighbour rows
        size += (36 + 4) * clusters + 6 * 401 * 4 + (16 + 4) * tracklets + (40 + 4) * cells + 4 * links
    pairs = tracklets * (tracklets / 6) / max(1.0, clusters / 7)  # per middle cluster: incoming times outgoing
    return size, 30 * clusters + 40 * tracklets + 10 * pairs + 60 * cells


def work(case):
    kind = case["kind"]
    if kind == "clustering":
        clusters = 7.2 * case["tracks"] * 1.05
        return {"bytes": 72 * clusters + 6 * 401 * 4, "flops": 30 * clusters}
    if kind == "train":
        n = case["samples"] + case["steps"] * case["batch"]
        return {"bytes": 33 * n + case["steps"] * 12 * capi.MLP_PARAMS, "flops": 6 * n * (8 * 64 + 64 * 64 + 64)}
    noise = 1.0 + case.get("noise", 0.10 if kind == "frames" else 0.05)
    if kind == "frames":
        runs = case["calls"] * case["frames"] * case["collisions"]
        clusters = 7.2 * case["tracks"] * noise * case["collisions"]
        size, flops = _event_work(case["tracks"], clusters, 36 / case["collisions"], collisions=case["collisions"])
        return {"bytes": runs * size, "flops": runs * flops}
    lo, hi, count = case["tracks"], case.get("tracks_max", case["tracks"]), case.get("events", 1)
    mults = [lo] if lo == hi else np.exp(np.linspace(math.log(lo), math.log(hi), 64))
    each = [_event_work(n, 7.2 * n * noise, 16 if kind == "stream" else 36, kind != "stream") for n in mults]
    return {"bytes": count * float(np.mean([w[0] for w in each])), "flops": count * float(np.mean([w[1] for w in each]))}


# ---- the same in 64 bits ----


def _exact_clustering(case, seed):
    """phi and r of every cluster in 64 bits, in the order of the sorted records: stable by bin, the bin
    from binary32 values as the index table's definition has it."""
    ev = gen.make_event(seed * SEED_STRIDE, case["tracks"])
    f, pi, two_pi = np.float32, np.float32(3.14159265359), np.float32(2.0) * np.float32(3.14159265359)
    half = (16.333, 16.333, 16.333, 42.140, 42.140, 73.745, 73.745)
    phis, rs = [], []
    for layer, c in enumerate(ev.layers):
        dx, dy = c["x"] - ev.vertices[0][0], c["y"] - ev.vertices[0][1]
        phi32 = np.arctan2(-dy.astype(np.float64), -dx.astype(np.float64)).astype(f) + pi
        phi32 = np.where(phi32 < 0, phi32 + two_pi, np.where(phi32 > two_pi, phi32 - two_pi, phi32))
        z_bin = ((c["z"] + f(half[layer])) * f(0.5 * 20 / float(f(half[layer])))).astype(np.int32)
        order = np.argsort(np.minimum((phi32 * (f(20) / two_pi)).astype(np.int32) * 20 + z_bin, 400), kind="stable")
        x, y = (c[k].astype(np.float64)[order] - float(v) for k, v in zip("xy", ev.vertices[0]))
        phis.append(np.arctan2(-y, -x) + math.pi)
        rs.append(np.hypot(x, y))
    room = np.zeros(_cluster_capacity(case["tracks"]) - sum(len(c) for c in ev.layers))  # behind the last cluster
    return {"sorted": None, "tables": None, "phi": np.concatenate(phis + [room]), "r": np.concatenate(rs + [room])}


def _exact_train(case, seed):
    """The full-set loss and gradient in 64 bits (no BF16 rounding); the minibatches of the Adam steps
    are drawn inside the library, so the trained parameters have no such value."""
    model = capi.prefilter_load(prefilter.CHECKPOINTS["pbpb"])
    features, labels = _samples(case, seed, model)
    x = (features.double() - torch.tensor(list(model.mean)).double()) * torch.tensor(list(model.inv_std)).double()
    params = {k: torch.from_numpy(np.asarray(model.arrays()[k], np.float64)).requires_grad_() for k in ("w1", "b1", "w2", "b2", "w3", "b3")}
    h = torch.nn.functional.gelu(x @ params["w1"].T + params["b1"], approximate="tanh")
    h = torch.nn.functional.gelu(h @ params["w2"].T + params["b2"], approximate="tanh")
    loss = torch.nn.functional.binary_cross_entropy_with_logits(h @ params["w3"] + params["b3"], labels.double())
    loss.backward()
    grad = torch.cat([params[k].grad.reshape(-1) for k in ("w1", "b1", "w2", "b2", "w3", "b3")])
    return {"grad": grad, "loss": float(loss.detach()), "losses": None, "params": None}


def exact(case, seed):
    if case["kind"] == "clustering":
        return _exact_clustering(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None  # record words: compared byte for byte
