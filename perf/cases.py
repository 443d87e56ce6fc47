"""Performance cases of the NRRS step: what a program has this library do, through the calls it
makes (nrrs_b200), at the sizes of the workloads in bench.py and tests/ and between them.

A renderer keeps one network context for its frame size. Per bounce it runs the RRS step on the
wavefront queue (inference, decision, next queue), from the full frame down to the last bounces'
few thousand vertices, or all depths in one captured graph. Per training frame it records path
nodes, builds the batch and takes training steps; the frame itself is traced and shaded around
the step. Every path exists in FP32, FP16 and BF16, for the 64- and 128-wide networks and for the
reference's shipped 32-wide one.

listed() and draw() give the cases, prepare() and run() one pass of a case, work() the bytes and
operations it cannot do without, exact() its outputs in 64 bits with plain torch."""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "nrrs-code_b200"))
import nrrs_b200 as nb  # noqa: E402

PREC = {"fp32": nb.PREC_FP32, "fp16": nb.PREC_FP16, "bf16": nb.PREC_BF16}
NETS = {"64x2": (64, 2), "64x3": (64, 3), "128x3": (128, 3), "shipped": (32, 3)}
TUNE_N = 1 << 20          # vertices of the tuning run a program makes once at start-up


def listed():
    return [
        # a late bounce of a 1080p frame, or a small preview tile: a few thousand vertices
        {"name": "step_tail_fp16", "kind": "step", "net": "64x2", "prec": "fp16", "log2": 19,
         "n": 3071, "max_queue": 2073600, "source": 3},
        # the plain FP32 step of 65,536 vertices
        {"name": "step_65536_fp32", "kind": "step", "net": "64x2", "prec": "fp32", "log2": 19,
         "n": 65536, "max_queue": 65536, "source": 3},
        # one full bounce of a 1920x1080 frame
        {"name": "step_1080p_fp16", "kind": "step", "net": "64x2", "prec": "fp16", "log2": 19,
         "n": 2073600, "max_queue": 2073600, "source": 3},
        # one full bounce of a 3840x2160 frame with the wide networks and the large table
        {"name": "step_4k_bf16", "kind": "step", "net": "128x3", "prec": "bf16", "log2": 22,
         "n": 8294400, "max_queue": 8294400, "source": 3},
        # all depths of a 1080p frame as one captured graph
        {"name": "graph_10_depths_fp16", "kind": "batched", "net": "64x2", "prec": "fp16",
         "log2": 19, "n": 2073600, "depths": 10, "source": 3},
        # the reference's shipped network on an odd queue of about 1280x720
        {"name": "step_720p_shipped_fp16", "kind": "step", "net": "shipped", "prec": "fp16",
         "log2": 19, "n": 921601, "max_queue": 2073600, "source": 3},
        # one training step of the 1080p frame
        {"name": "train_262144_fp16", "kind": "train", "net": "64x2", "prec": "fp16", "log2": 19,
         "n": 262144},
        # one training step of the 4K frame
        {"name": "train_262144_bf16_128x3", "kind": "train", "net": "128x3", "prec": "bf16",
         "log2": 22, "n": 262144},
        # the plain FP32 training step
        {"name": "train_262144_fp32", "kind": "train", "net": "64x2", "prec": "fp32", "log2": 19,
         "n": 262144},
        # the shipped network on a ragged path-record batch with its per-sample loss inputs
        {"name": "train_batch_50021_shipped", "kind": "train_batch", "net": "shipped",
         "prec": "fp16", "log2": 19, "n": 50021},
        # the training side of a 1280x720 frame: records, radiance, batch, weights
        {"name": "records_720p", "kind": "records", "pixels": 921600, "bounces": 6},
        # a 1280x720 frame traced and shaded around the step, three bounces
        {"name": "render_720p_fp16", "kind": "render", "net": "64x2", "prec": "fp16", "log2": 19,
         "width": 1280, "height": 720, "bounces": 3, "boxes": 1000},
    ]


def draw(rng):
    def size(lo, hi):
        v = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
        return v | 1 if rng.random() < 0.5 else v

    u = rng.random()
    if u < 0.45:
        prec = rng.choice(["fp32", "fp16", "fp16", "bf16"])
        net = rng.choice(["64x2", "64x2", "64x3", "128x3", "shipped"])
        n = size(1000, 500000 if prec == "fp32" else 4000000)
        return {"kind": "step", "net": net, "prec": prec,
                "log2": 22 if net == "128x3" and rng.random() < 0.3 else 19, "n": n,
                "max_queue": max(n, rng.choice([65536, 921600, 2073600])),
                "source": rng.choice([3, 3, 3, 2])}
    if u < 0.55:
        return {"kind": "batched", "net": rng.choice(["64x2", "64x3"]),
                "prec": rng.choice(["fp16", "bf16"]), "log2": 19, "n": size(20000, 2000000),
                "depths": rng.randint(2, 12), "source": 3}
    if u < 0.77:
        return {"kind": "train", "net": rng.choice(["64x2", "64x3", "128x3"]),
                "prec": rng.choice(["fp32", "fp16", "bf16"]), "log2": 19, "n": size(2000, 262144)}
    if u < 0.87:
        return {"kind": "train_batch", "net": rng.choice(["shipped", "64x2"]),
                "prec": rng.choice(["fp32", "fp16"]), "log2": 19, "n": size(2000, 200000)}
    if u < 0.94:
        return {"kind": "records", "pixels": size(20000, 1500000), "bounces": rng.randint(3, 8)}
    h = rng.randint(90, 800)
    return {"kind": "render", "net": "64x2", "prec": "fp16", "log2": 19, "width": h * 16 // 9,
            "height": h, "bounces": rng.randint(2, 4), "boxes": rng.randint(40, 1500)}


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)


def _unit(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda")
    return (v / v.norm(dim=1, keepdim=True).clamp_min(1e-20)).contiguous()


def _vertices(seed, n, target=False):
    """Vertices with the distributions of the library's synthetic queue (csrc/synth.cpp)."""
    g = _gen(seed, 1)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda")      # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")    # noqa: E731
    v = {"pos": rand(n, 3), "wi": _unit(g, n), "normal": _unit(g, n), "roughness": rand(n),
         "albedo": rand(n, 3), "thp": torch.exp(randn(n, 3) - 1.0),
         "depth": (rand(n) * 6.0).to(torch.int32).clamp_(max=5),
         "ref_mean": torch.exp(randn(n) - 1.0), "rnd": rand(n)}
    if target:
        t = torch.exp(2.0 * randn(n, 3))
        v["target"] = t * torch.where(rand(n) < 0.01, 100.0, 1.0)[:, None]
    return v


def _soa(v, **more):
    return nb.vertex_soa(v["pos"], v["wi"], v["normal"], v["roughness"], v["albedo"], v["thp"],
                         v["depth"], v.get("ref_mean"), **more)


class Shape:
    """The level table and the layer shapes of a case's networks (include/nrrs.h)."""

    def __init__(self, case):
        self.shipped = case["net"] == "shipped"
        self.width, self.hidden = NETS[case["net"]]
        self.levels, scale = (8, 2.0) if self.shipped else (16, 1.5)
        T, off, self.level = 1 << case["log2"], 0, []
        for i in range(self.levels):
            res = int(math.floor(16 * scale ** i))
            dense = (res + 1) ** 3 <= T
            self.level.append((res, dense, off))
            off += (res + 1) ** 3 if dense else T
        self.rows, self.mask = off, T - 1
        self.sin, self.sout = (32, 6) if self.shipped else (64, 3)

        def layers(k, out):
            w = self.width
            return [(w, k)] + [(w, w)] * (self.hidden - 1) + [(out, w)]

        self.stat, self.rrs = layers(self.sin, self.sout), layers(16, 1)
        self.mlp = sum(o * k for o, k in self.stat + self.rrs)
        self.params = 2 * self.rows + self.mlp


def _params(case, seed):
    """Weights as training leaves them: features of a few tenths, Xavier-sized layers."""
    s, g = Shape(case), _gen(seed, 2)
    parts = [0.2 * torch.randn(2 * s.rows, generator=g, device="cuda")]
    for o, k in s.stat + s.rrs:
        a = math.sqrt(6.0 / (o + k))
        parts.append((torch.rand(o * k, generator=g, device="cuda") * 2.0 - 1.0) * a)
    return torch.cat(parts)


def _config(case, **kw):
    w, h = NETS[case["net"]]
    kw.update(precision=PREC[case["prec"]], log2_hashmap_size=case["log2"])
    if case["net"] == "shipped":
        return nb.reference_config(**kw)
    return nb.default_config(statnet_width=w, statnet_hidden=h, rrsnet_width=w, rrsnet_hidden=h,
                             **kw)


def _network(case, seed, tune=True, **kw):
    net = nb.NRRSNetwork(_config(case, **kw))
    net.set_params(_params(case, seed).cpu().numpy())
    if tune and case["prec"] != "fp32":
        net.autotune(min(TUNE_N, net.config.max_queue))
    return net


def _step_out(case, n, cap, sizes=1):
    z = lambda n, t=torch.float32: torch.zeros(n, dtype=t, device="cuda")   # noqa: E731
    return {"stats": z((n, Shape(case).sout)), "rrs": z(n), "rrs_norm": z(n),
            "split": z(n, torch.uint8), "queue": z(cap, torch.int32), "size": z(sizes, torch.int32)}


def _segments(case):
    """Vertices per depth: 0.6 of the depth before, a tenth of them split into 1 to 4."""
    return [max(1, int(round(case["n"] * 0.6 ** d * 1.15))) for d in range(case["depths"])]


# ---- the cases' passes --------------------------------------------------------------------------

def prepare(case, seed):
    state = {"step": _prepare_step, "batched": _prepare_batched, "train": _prepare_train,
             "train_batch": _prepare_train_batch, "records": _prepare_records,
             "render": _prepare_render}[case["kind"]](case, seed)
    state["stream"] = torch.cuda.current_stream().cuda_stream
    return state


def run(state):
    return state["pass"](state)


def _prepare_step(case, seed):
    n, cap = case["n"], 2 * case["n"] + 1024
    s = {"pass": _run_step, "n": n, "cap": cap, "v": _vertices(seed, n),
         "out": _step_out(case, n, cap), "dp": nb.default_decide(factor_source=case["source"]),
         "net": _network(case, seed, max_queue=case["max_queue"], max_train=1024)}
    s["soa"] = _soa(s["v"])
    return s


def _run_step(s):
    o, n = s["out"], s["n"]
    s["net"].generateRRSNumber(s["soa"], s["v"]["rnd"], n, n, 0, s["dp"], o["stats"], o["rrs"],
                               o["rrs_norm"], o["split"], o["queue"], s["cap"], o["size"],
                               s["stream"])
    return o


def _prepare_batched(case, seed):
    counts = _segments(case)
    n = sum(counts)
    segs, off, qoff = [], 0, 0
    for c in counts:
        segs.append(nb.Segment(off, c, c, 0, qoff, 2 * c + 1024))
        off, qoff = off + c, qoff + 2 * c + 1024
    s = {"pass": _run_batched, "v": _vertices(seed, n), "out": _step_out(case, n, qoff, len(counts)),
         "dp": nb.default_decide(factor_source=case["source"]),
         "net": _network(case, seed, max_queue=n, max_train=1024)}
    s["soa"], o = _soa(s["v"]), s["out"]
    s["graph"] = s["net"].captureBatched(s["soa"], s["v"]["rnd"], segs, s["dp"], o["stats"],
                                         o["rrs"], o["rrs_norm"], o["split"], o["queue"],
                                         o["size"])
    return s


def _run_batched(s):
    s["graph"].launch(s["stream"])
    return s["out"]


def _train_out(case):
    """The gradient vector and a step's outputs: the losses and the vector's three groups."""
    s = Shape(case)
    g = torch.zeros(s.params, device="cuda")
    a, b = 2 * s.rows, 2 * s.rows + sum(o * k for o, k in s.stat)
    return g, {"loss": torch.zeros(2, dtype=torch.float64, device="cuda"), "table": g[:a],
               "statnet": g[a:b], "rrsnet": g[b:]}


LR = 1e-4    # a late step of the schedule, which a program can repeat for long


def _prepare_train(case, seed):
    n = case["n"]
    s = {"pass": _run_train, "n": n, "v": _vertices(seed, n, target=True),
         "net": _network(case, seed, tune=False, max_queue=1024, max_train=n, lr=LR)}
    s["grads"], s["out"] = _train_out(case)
    s["soa"] = _soa(s["v"])
    return s


def _run_train(s):
    s["net"].train(s["soa"], s["v"]["target"], s["n"], s["out"]["loss"], s["stream"])
    s["net"].copyGrads(s["grads"], s["stream"])     # kept by the program (norms, logs, all-reduce)
    return s["out"]


def _loss_inputs(seed, n, target):
    """The per-sample loss inputs of a path-record batch: pixel shares, RRSNet targets with the
    duplicate mark, pixel errors and sample counts; and the error image's sum."""
    g = _gen(seed, 3)
    u = torch.rand(n, 4, generator=g, device="cuda")
    k = torch.floor(1.0 + 3.0 * u[:, 0])
    return {"weight": (1.0 / k).contiguous(),
            "rrs_target": torch.where(u[:, 1] < 0.15, -1.0, 0.2 + 2.0 * u[:, 1]),
            "error": (2.0 * u[:, 2] ** 2).contiguous(),
            "error_for_avg": (2.0 * u[:, 2] ** 2 * k.sqrt()).contiguous(),
            "number_samples": k.contiguous(),
            "error_sum": torch.full((1,), 0.7 * 4096, device="cuda")}


GAMMAS = (1.0, 0.2, 0.1, 0.01)


def _prepare_train_batch(case, seed):
    n = case["n"]
    v = _vertices(seed, n, target=True)
    v["target"].clamp_(max=10.0)      # linear radiance statistics: the filtered batch's range
    side = _loss_inputs(seed, n, v["target"])
    kw = dict(lr=LR) if case["net"] != "shipped" else dict(lr=LR, lr_rrsnet=LR)
    s = {"pass": _run_train_batch, "n": n, "v": v, "side": side,
         "net": _network(case, seed, tune=False, max_queue=1024, max_train=n, **kw),
         "lp": nb.default_loss_params(gamma1=GAMMAS[0], gamma2=GAMMAS[1], gamma3=GAMMAS[2],
                                      gamma4=GAMMAS[3], clamp_on=1, clamp_max=10.0, n_pixels=4096)}
    s["grads"], s["out"] = _train_out(case)
    s["batch"] = nb.train_batch(
        **{k: v[k] for k in ("pos", "wi", "normal", "albedo", "roughness", "thp", "depth",
                             "ref_mean", "target")},
        **{k: side[k] for k in ("rrs_target", "error", "error_for_avg", "number_samples")})
    return s


def _run_train_batch(s):
    s["net"].trainStepBatch(s["batch"], s["n"], s["side"]["weight"], s["side"]["error_sum"],
                            s["lp"], s["out"]["loss"], s["stream"])
    s["net"].copyGrads(s["grads"], s["stream"])
    return s["out"]


BATCH_F = {"pos": 3, "wi": 3, "normal": 3, "albedo": 3, "roughness": 1, "thp": 3, "ref_mean": 1,
           "target": 3, "rrs_target": 1}


def _paths(case, seed):
    """A training frame's bounces, as synth_paths draws them, made on the device; its nodes."""
    g = _gen(seed, 4)
    pix = torch.arange(case["pixels"], device="cuda")
    parent = torch.full((case["pixels"],), -1, device="cuda")
    thp_prev = torch.ones(case["pixels"], 3, device="cuda")
    out, nodes = [], 0
    for d in range(case["bounces"]):
        n = pix.numel()
        r = torch.rand(n, 16, generator=g, device="cuda")
        rec = r[:, 0] < 0.7
        node = torch.where(rec, nodes + torch.cumsum(rec, 0) - 1, parent)
        nodes += int(rec.sum())
        thp = (thp_prev * (0.3 + 0.7 * r[:, 1:4])).contiguous()
        k = (r[:, 4] >= 0.4).long() + (r[:, 4] >= 0.85).long()
        src = torch.repeat_interleave(torch.arange(n, device="cuda"), k)
        le = torch.exp(1.5 * torch.randn(src.numel(), 3, generator=g, device="cuda"))
        le *= (torch.rand(src.numel(), 1, generator=g, device="cuda") >= 0.1)
        out.append({"pos": r[:, 5:8].contiguous(), "wi": _unit(g, n), "normal": _unit(g, n),
                    "albedo": r[:, 8:11].contiguous(), "roughness": r[:, 11].contiguous(),
                    "thp": thp, "depth": torch.full((n,), d, dtype=torch.int32, device="cuda"),
                    "pixel": pix.int(), "rrs": (0.2 + 2.8 * r[:, 12]).contiguous(),
                    "record": rec.to(torch.uint8), "parent": parent.int(),
                    "contrib_node": node[src].int().contiguous(),
                    "contrib": (thp[src] * le).contiguous(),
                    "node_out": torch.zeros(n, dtype=torch.int32, device="cuda")})
        s = (r[:, 13] >= 0.35).long() + (r[:, 13] >= 0.85).long() + (r[:, 13] >= 0.95).long()
        nxt = torch.repeat_interleave(torch.arange(n, device="cuda"), s)
        pix, parent, thp_prev = pix[nxt], node[nxt], thp[nxt]
    image = 2.0 * torch.rand(case["pixels"], 4, generator=g, device="cuda")
    return out, nodes, image


def _prepare_records(case, seed):
    P = case["pixels"]
    bounces, nodes, image = _paths(case, seed)
    # the reference sizes its node buffer per pixel (10 at 8 bounces) and never grows it
    cap = int(P * (case["bounces"] + 2))
    most = max(b["pixel"].numel() for b in bounces)
    nbytes = nb.path_nodes_bytes(cap, most)
    block = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    z = lambda *s, t=torch.float32: torch.zeros(*s, dtype=t, device="cuda")   # noqa: E731
    # the batch arrays hold a sample per pixel and bounce: more than 0.7 of a shrinking queue
    most_t = P * case["bounces"]
    batch = {k: z(most_t, 3) if w == 3 else z(most_t) for k, w in BATCH_F.items()}
    batch["depth"], batch["pixel"] = z(most_t, t=torch.int32), z(most_t, t=torch.int32)
    s = {"pass": _run_records, "bounces": bounces, "image": image, "P": P, "most": most_t,
         "block": block, "counts": z(P, t=torch.int32),
         "out": dict(batch, size=z(1, t=torch.int32), weight=z(most_t)),
         "prm": nb.default_train_data_params(copy_rrs_node=1, dedupe_rrs_target=1,
                                             frame_width=P),
         "buf": nb.NRRSPathNodesBuffer(block.data_ptr(), nbytes, cap, most)}
    s["batch"] = nb.train_batch(**batch)
    for b in bounces:
        b["soa"] = _soa(b)
    return s


def _run_records(s):
    buf, st, o = s["buf"], s["stream"], s["out"]
    buf.reset(st)
    for b in s["bounces"]:
        buf.recordNode(b["soa"], b["parent"], b["pixel"], b["rrs"], b["record"],
                       b["pixel"].numel(), b["node_out"], st)
        buf.recordRadiance(b["contrib_node"], b["contrib"], b["contrib_node"].numel(), st)
    s["counts"].zero_()
    buf.generate_training_data(s["prm"], s["batch"], s["most"], o["size"], image=s["image"],
                               n_pixels=s["P"], pixel_samples=s["counts"], stream=st)
    nb.calculate_sample_weight(o["pixel"], s["counts"], s["P"], o["size"], s["most"],
                               o["weight"], st)
    return o


def _prepare_render(case, seed):
    P = case["width"] * case["height"]
    cap = 3 * P
    scene = nb.Scene(*nb.synth_scene(seed % 1000, n_boxes=case["boxes"], closed=True))
    f = lambda *s: torch.zeros(*s, dtype=torch.float32, device="cuda")   # noqa: E731
    i = lambda *s: torch.zeros(*s, dtype=torch.int32, device="cuda")     # noqa: E731
    rays = {"origin": f(cap, 3), "dir": f(cap, 3), "thp": f(cap, 3), "pdf": f(cap),
            "pixel": i(cap), "node": i(cap)}
    hits = {"prim": i(cap), "t": f(cap), "u": f(cap), "v": f(cap)}
    verts = {"pos": f(cap, 3), "wi": f(cap, 3), "normal": f(cap, 3), "albedo": f(cap, 3),
             "roughness": f(cap), "thp": f(cap, 3), "depth": i(cap), "pixel": i(cap),
             "node": i(cap)}
    shadow = {"origin": f(cap, 3), "dir": f(cap, 3), "tmax": f(cap), "contrib": f(cap, 3),
              "pixel": i(cap), "node": i(cap)}
    s = {"pass": _run_render, "scene": scene, "P": P, "cap": cap, "bounces": case["bounces"],
         "cam": nb.room_camera(case["width"], case["height"], inside=True), "seed": seed & 0xFFFF,
         "net": _network(case, seed, max_queue=cap, max_train=1024),
         # an untrained network: factors of at least 1 keep about one path per pixel
         "dp": nb.default_decide(clamp_min=1.0),
         "bufs": (rays, hits, verts, shadow), "film": torch.zeros(P, 9, dtype=torch.int64, device="cuda"),
         "R": nb.soa(nb.RaySoA, rays), "H": nb.soa(nb.HitSoA, hits),
         "V": nb.soa(nb.PathVertices, verts), "S": nb.soa(nb.ShadowSoA, shadow), "vsoa": _soa(verts),
         "scr": torch.zeros(nb.shade_scratch_bytes(cap), dtype=torch.uint8, device="cuda"),
         "tscr": torch.zeros(nb.trace_scratch_bytes(cap), dtype=torch.uint8, device="cuda"),
         "rnd": torch.rand(cap, generator=_gen(seed, 5), device="cuda"), "n_rays": i(1),
         "stats": f(cap, 3), "split": torch.zeros(cap, dtype=torch.uint8, device="cuda"),
         "queue": i(cap), "rrs_norm": f(cap),
         "out": {"image": f(P, 3), "rrs": f(cap), "vertices": i(1), "size": i(1)}}
    return s


def _run_render(s):
    st, o, sc, cap, P = s["stream"], s["out"], s["scene"], s["cap"], s["P"]
    s["film"].zero_()
    nb.camera_rays(s["cam"], 0, s["seed"], s["R"], st)
    s["n_rays"].fill_(P)
    for d in range(s["bounces"]):
        if d == 0:
            nb.trace(sc, s["R"], s["n_rays"], cap, s["H"], st)
        else:
            nb.trace_sorted(sc, s["R"], s["n_rays"], cap, s["H"], s["tscr"], st)
        nb.shade(sc, s["R"], s["H"], s["n_rays"], cap, d, s["film"], None, s["V"], o["vertices"],
                 s["scr"], st)
        s["net"].generateRRSNumberDev(s["vsoa"], s["rnd"], o["vertices"], cap, P, 0, s["dp"],
                                      s["stats"], o["rrs"], s["rrs_norm"], s["split"], s["queue"],
                                      cap, o["size"], stream=st)
        nb.scatter(sc, s["V"], s["rrs_norm"], s["queue"], o["size"], cap, d, s["seed"], s["R"],
                   s["S"], st)
        nb.trace_shadow(sc, s["S"], o["size"], cap, s["film"], None, st)
        s["n_rays"].copy_(o["size"])
    nb.film_resolve(s["film"], P, 1.0, o["image"], st)
    return o


# ---- work ---------------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "records":
        # vertices shrink by 0.85 a bounce, 0.7 of them record, 0.75 contributions each
        v = case["pixels"] * sum(0.85 ** d for d in range(case["bounces"]))
        return {"bytes": v * (85 + 16 * 0.75 + 4) + 0.7 * v * (84 + 100) + 28 * case["pixels"],
                "flops": 0}
    s = Shape(case)
    flop = 2 * s.mlp + 16 * 2 * s.levels
    byte = 4 if case["prec"] == "fp32" else 2
    if kind in ("train", "train_batch"):
        n = case["n"]
        side = 24 if kind == "train_batch" else 0
        # inputs, the table's touched rows, gradients out (and kept), Adam on every parameter
        return {"bytes": n * (84 + side) + min(2 * s.rows * byte, n * s.levels * 16 * byte) +
                s.params * (8 + 24), "flops": 3 * flop * n}
    if kind == "render":
        n = case["width"] * case["height"] * case["bounces"]
        ray = 44 + 12 + 16 + 76 + 44 + 40
        return {"bytes": n * (ray + 101) + 84 * case["width"] * case["height"], "flops": flop * n}
    n = sum(_segments(case)) if kind == "batched" else case["n"]
    return {"bytes": n * (76 + 13 + 4 * s.sout + 4) +
            min(2 * s.rows * byte, n * s.levels * 16 * byte) + s.mlp * byte, "flops": flop * n}


# ---- the same outputs in 64 bits ----------------------------------------------------------------

def _layers64(case, seed):
    s, p = Shape(case), _params(case, seed)
    table, at = p[:2 * s.rows].view(-1, 2), 2 * s.rows
    nets = []
    for shapes in (s.stat, s.rrs):
        w = []
        for o, k in shapes:
            w.append(p[at:at + o * k].view(o, k).double())
            at += o * k
        nets.append(w)
    return s, table, nets[0], nets[1]


def _hash64(s, pos, table):
    """The grid's features of positions in [0, 1]; table [rows, 2]."""
    p, out = pos.double().clamp(0.0, 1.0), []
    for res, dense, off in s.level:
        x = p * res
        c = x.floor().clamp(0, res - 1)
        f, c = x - c, c.long()
        acc = 0.0
        for k in range(8):
            b = [(k >> j) & 1 for j in range(3)]
            g = [c[:, j] + b[j] for j in range(3)]
            if dense:
                i = g[0] + (res + 1) * (g[1] + (res + 1) * g[2])
            else:
                i = (g[0] ^ (g[1] * 2654435761) ^ (g[2] * 805459861)) & s.mask
            w = 1.0
            for j in range(3):
                w = w * (f[:, j] if b[j] else 1.0 - f[:, j])
            acc = acc + w[:, None] * table[off + i].double()
        out.append(acc)
    return torch.cat(out, 1)


def _sh64(d):
    x, y, z = d.double().unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    pi = math.pi
    a, b = math.sqrt(3 / (4 * pi)), math.sqrt(15 / (4 * pi))
    c = [torch.full_like(x, 0.5 / math.sqrt(pi)), -a * y, a * z, -a * x,
         b * x * y, -b * y * z, math.sqrt(5 / (16 * pi)) * (3 * zz - 1), -b * x * z,
         0.5 * b * (xx - yy)]
    e, f = math.sqrt(35 / (32 * pi)), math.sqrt(105 / (4 * pi))
    g, h = math.sqrt(21 / (32 * pi)), math.sqrt(7 / (16 * pi))
    c += [-e * y * (3 * xx - yy), f * x * y * z, -g * y * (5 * zz - 1), h * z * (5 * zz - 3),
          -g * x * (5 * zz - 1), 0.5 * f * z * (xx - yy), -e * x * (xx - 3 * yy)]
    return torch.stack(c, 1)


def _blob64(x, bins):
    k = torch.arange(bins + 1, device=x.device, dtype=torch.float64) / bins
    u = ((k[None, :] - x[:, None]) * bins).clamp(-1, 1)
    cdf = 15 / 16 * u * (1 - 2 / 3 * u ** 2 + u ** 4 / 5) + 0.5
    return cdf[:, 1:] - cdf[:, :-1]


def _mlp64(x, w, shipped):
    for m in w[:-1]:
        x = x @ m.t()
        x = torch.where(x > 0, x, 0.01 * x) if shipped else x.relu()
    return x @ w[-1].t()


def _statnet64(s, v, table, w):
    warp = 1 - torch.exp(-v["roughness"].double())
    grid = _hash64(s, v["pos"], table)
    if s.shipped:
        d = v["wi"].double()
        u = torch.atan2(d[:, 1], d[:, 0]) / (2 * math.pi) + 0.5
        t = torch.acos(d[:, 2].clamp(-1, 1)) / math.pi
        x = torch.cat([grid, _blob64(u, 4), _blob64(t, 4), _blob64(warp, 8)], 1)
    else:
        one = torch.ones_like(warp)[:, None]
        x = torch.cat([grid, _sh64(v["wi"]), v["normal"].double(), v["albedo"].double(),
                       warp[:, None], one, one.new_zeros(one.shape[0], 8)], 1)
    return _mlp64(x, w, s.shipped)


def _bc64(x):
    return 2 * (x.sqrt() - 1)


def _rrsnet64(s, v, y, w):
    warp = 1 - torch.exp(-v["roughness"].double())
    thp, ref = v["thp"].double(), v["ref_mean"].double()
    one = torch.ones_like(warp)
    if s.shipped:
        x = torch.cat([_bc64(y.clamp_min(0)), _bc64(thp),
                       torch.stack([warp, _bc64(ref), one], 1), one.new_zeros(len(one), 4)], 1)
    else:
        lum = (torch.exp(y.clamp_max(20)) - 0.01).clamp_min(0)
        x = torch.cat([_bc64(lum), _bc64(thp),
                       torch.stack([warp, _bc64(ref), v["depth"].double() / 8, one], 1),
                       one.new_zeros(len(one), 6)], 1)
    raw = _mlp64(x, w, s.shipped)[:, 0]
    return raw, torch.where(raw < 0, torch.log1p(torch.exp(raw.clamp_max(0))),
                            0.5 * raw + math.log(2.0))


def _cut(v, a, b):
    return {k: t[a:b] for k, t in v.items()}


def _exact_step(case, seed, counts):
    s, table, ws, wr = _layers64(case, seed)
    v = _vertices(seed, sum(counts))
    stats, rrs = [], []
    for a in range(0, sum(counts), 1 << 18):
        c = _cut(v, a, a + (1 << 18))
        y = _statnet64(s, c, table, ws)
        if case["source"] == nb.FACTOR_ADRRS:
            lum = y[:, :3] if s.shipped else torch.exp(y.clamp_max(20)) - 0.01
            q = (lum.clamp(1e-4, 1e4) * c["thp"].double()).mean(1) / (c["ref_mean"].double() + 0.01)
        else:
            q = _rrsnet64(s, c, y, wr)[1]
        stats.append(y)
        rrs.append(q.clamp(float(np.float32(0.05)), 8.0))
    rrs, norm, a = torch.cat(rrs), [], 0
    for n in counts:
        r = rrs[a:a + n]
        norm.append(r * min(float(n / r.ceil().sum()), 1.0))
        a += n
    return {"stats": torch.cat(stats), "rrs": rrs, "rrs_norm": torch.cat(norm), "split": None,
            "queue": None, "size": None}


def _exact_train(case, seed):
    s, table, ws, wr = _layers64(case, seed)
    n = case["n"]
    v = _vertices(seed, n, target=True)
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    sw, var, cost, reg = one, one, one, 0 * one      # per-sample weights of the losses' terms
    if case["kind"] == "train_batch":
        v["target"].clamp_(max=10.0)
        side = {k: t.double() for k, t in _loss_inputs(seed, n, v["target"]).items()}
        mean = float(side["error_sum"][0]) / 4096
        sw = side["weight"]
        w = torch.where(side["rrs_target"] < 0, 0 * sw, sw)
        u = GAMMAS[0] + sum(g * (side[k] / mean).clamp_max(10.0)
                            for g, k in zip(GAMMAS[1:3], ("error", "error_for_avg")))
        cost = w * (n / w.sum())
        var = cost * u / side["number_samples"].clamp_min(1)
        reg, sw = GAMMAS[3] * cost, sw * (n / sw.sum())
    lum = v["target"].double()
    r = ((v["thp"].double() * lum).mean(1) / (v["ref_mean"].double() + 0.01)).clamp_max(10.0)
    step, ys = 1 << 15, []
    sumV = sumC = sumR = lossS = 0.0
    for a in range(0, n, step):
        c, i = _cut(v, a, a + step), slice(a, a + step)
        y = _statnet64(s, c, table, ws)
        q = _rrsnet64(s, c, y, wr)[1]
        sumV += float((var[i] * r[i] ** 2 / q).sum()) / n
        sumC += float((cost[i] * (1 + q)).sum()) / n
        sumR += float((reg[i] * q.log() ** 2).sum()) / n
        ys.append(y)
    gt = torch.zeros(s.rows, 2, dtype=torch.float64, device="cuda")
    table = table.double().requires_grad_()
    weights = [m.requires_grad_() for m in ws + wr]
    for a in range(0, n, step):
        c, i = _cut(v, a, a + step), slice(a, a + step)
        y = _statnet64(s, c, table, ws)
        if s.shipped:
            t = torch.cat([lum[i], lum[i] ** 2], 1)
            e = (y - t) ** 2 / (t * t + 0.01)
        else:
            e = (y - torch.log(lum[i] + 0.01)) ** 2
        loss = (sw[i, None] * e).sum() / (s.sout * n)
        lossS += float(loss.detach())
        q = _rrsnet64(s, c, ys[a // step], wr)[1]
        loss = loss + (var[i] * r[i] ** 2 / q).sum() / n * sumC + (cost[i] * q).sum() / n * sumV \
            + (reg[i] * q.log() ** 2).sum() / n
        loss.backward()
        gt += table.grad
        table.grad = None
    return {"loss": torch.tensor([lossS, sumV * sumC + sumR], dtype=torch.float64),
            "table": gt.view(-1), "statnet": torch.cat([m.grad.reshape(-1) for m in ws]),
            "rrsnet": torch.cat([m.grad.reshape(-1) for m in wr])}


def _exact_records(case, seed):
    bounces, nodes, image = _paths(case, seed)
    rad = torch.zeros(nodes, 3, dtype=torch.float64, device="cuda")
    thp, rrs, pix, spans, at = [], [], [], [], 0
    for b in bounces:
        ok = b["contrib_node"] >= 0
        rad.index_add_(0, b["contrib_node"][ok].long(), b["contrib"][ok].double())
        m = b["record"].bool()
        spans.append((at, at + int(m.sum()), b["parent"][m].long()))
        at = spans[-1][1]
        thp.append(b["thp"][m].double())
        rrs.append(b["rrs"][m].double())
        pix.append(b["pixel"][m].long())
    for a, z, parent in reversed(spans):
        ok = parent >= 0
        rad.index_add_(0, parent[ok], rad[a:z][ok])
    thp, rrs = torch.cat(thp), torch.cat(rrs)
    out = {k: None for k in list(BATCH_F) + ["depth", "pixel", "size", "weight"]}
    out["target"] = torch.where(thp > 1e-5, rad / thp, 0 * rad)
    out["thp"] = thp * rrs[:, None]
    out["ref_mean"] = image[torch.cat(pix), :3].double().mean(1)
    for k in ("target", "thp", "ref_mean"):      # the arrays' unused rest
        rest = out[k].new_zeros((case["pixels"] * case["bounces"] - nodes,) + out[k].shape[1:])
        out[k] = torch.cat([out[k], rest])
    return out


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "step":
            return _exact_step(case, seed, [case["n"]])
        if case["kind"] == "batched":
            return _exact_step(case, seed, _segments(case))
        if case["kind"] == "records":
            return _exact_records(case, seed)
    if case["kind"] in ("train", "train_batch"):
        return _exact_train(case, seed)
    return None      # a path-traced frame: its brute-force trace takes minutes
