"""The workloads this framework is measured on: whole passes through ``SpDNN`` (set an input, run the layer loop, fetch
the surviving images), as the drivers, the benchmark and a serving program make them.

Sizes are those of the challenge networks (N = 1024, 4096, 16384, 65536 neurons; 120, 480, 1920 layers; batches up to
60000 images) and of small and ragged batches of the same networks.  ``net`` names the network:

  radix16  32 inputs per neuron, all weights 1/16, butterfly of 16-wide blocks (what the challenge networks are)
  random   32 inputs per neuron drawn at random, all weights 1/16, every layer another matrix (no structure to use)
  general  20 or 37 inputs per neuron with a tenth of them missing, every weight another value

``input`` names how the images reach the library:

  dense_device  fp32 matrix on the GPU              dense_host  the same in pageable host memory
  bits_device   bit matrix on the GPU               bits_host   the same in page-locked host memory
  coo_host      (image, neuron) triplets in host memory, the form of the challenge's input files

``images``: "blobs" are binary, three discs per image, 15 % of the pixels set; "mixed" are binary without spatial
structure, 5 to 60 % set (what survives in networks without locality); "grey" are blobs of intensities in [0.5, 2).
``fetch``: "ids" = the category list and the per-layer live counts, "all" = the survivors' activations too.
``slices`` > 1: the batch goes through two contexts in turn, so that one slice's copy overlaps the other's layers."""
import ctypes
import math

import numpy as np
import torch

from graphchallenge21_b200 import SpDNN
from graphchallenge21_b200.generator import SyntheticNetwork, rand_unit

PIXELS = (1024, 4096, 16384, 65536)
GENERAL_BIAS = -0.25


def _case(name, neurons, layers, batch, net="radix16", input="dense_device", images="blobs", fetch="ids", slices=1):
    c = {"neurons": neurons, "layers": layers, "batch": batch, "net": net, "input": input, "images": images, "fetch": fetch,
         "slices": slices}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one image through the smallest network: what an interactive caller waits for
        _case("one_image", 1024, 120, 1, input="dense_host"),
        # two tiles of images through a full-depth network: latency of the layer chain
        _case("few_images_deep", 16384, 1920, 64, input="bits_host"),
        # the network and batch of the drivers' usage example, in the input format the drivers read
        _case("driver_n1024", 1024, 120, 6000, input="coo_host"),
        # challenge networks at the full batch: N = 1024 from host memory, N = 4096 and 16384 from the GPU
        _case("full_n1024", 1024, 1920, 60000, input="bits_host"),
        _case("full_n4096", 4096, 480, 60000),
        _case("full_n16384", 16384, 1920, 60000),
        # the same batch served from host memory in slices, two contexts in turn
        _case("sliced_n16384", 16384, 1920, 60000, input="bits_host", slices=4),
        # the largest network, one GPU's share of the batch on eight
        _case("share_n65536", 65536, 1920, 7500, input="bits_device"),
        # inputs that are not binary, a ragged batch, activations wanted back
        _case("grey_n4096", 4096, 120, 5001, images="grey", fetch="all"),
        # no structure in the network: every output gathers 32 different rows
        _case("random_n1024", 1024, 120, 60000, net="random", images="mixed"),
        # the same where the activations of an image do not fit on the chip: one launch per layer
        _case("random_n16384", 16384, 24, 3000, net="random", images="mixed"),
        # general weights and ragged columns, activations wanted back
        _case("general_n1024", 1024, 24, 6000, net="general", images="mixed", fetch="all"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    net = rng.choice(["radix16"] * 5 + ["random", "general"])
    if net == "general":
        neurons = rng.choice([256, 512, 1024])
        return _case(None, neurons, rng.randint(4, 24), _log_int(rng, 1, 6000), net, rng.choice(["dense_device", "dense_host"]), "mixed",
                     rng.choice(["ids", "all"]))
    if net == "random":
        neurons = rng.choice([1024, 4096, 16384])
        layers = rng.randint(8, 120) if neurons == 1024 else rng.randint(4, 24)
        most = {1024: 60000, 4096: 12000, 16384: 3000}[neurons]
        return _case(None, neurons, layers, _log_int(rng, 1, most), net, rng.choice(["dense_device", "bits_device"]), "mixed")
    neurons = rng.choice(PIXELS)
    layers = _log_int(rng, 16, 1920)
    most = {1024: 60000, 4096: 60000, 16384: 60000, 65536: 7500}[neurons]
    batch = _log_int(rng, 1, most)
    if rng.random() < 0.2:
        return _case(None, neurons, layers, min(batch, 2 ** 25 // neurons), input=rng.choice(["dense_device", "dense_host"]), images="grey",
                     fetch=rng.choice(["ids", "all"]))
    form = rng.choice(["dense_device", "bits_device", "bits_host", "dense_host", "coo_host"])
    if form in ("dense_host", "coo_host"):
        batch = min(batch, 2 ** 26 // neurons)
    slices = rng.choice([1, 1, 2, 4]) if form == "bits_host" and batch >= 256 else 1
    return _case(None, neurons, layers, batch, input=form, slices=slices)


# ---- the network: a program loads it once, so its host form is kept from one preparation to the next --------------

_LAYERS = {}


def _general_layer(neurons, layer):
    rng = np.random.default_rng(1000 + layer)
    k = 20 if layer % 2 else 37
    # k distinct rows per column: one from each of k equal ranges of the rows
    edges = np.linspace(0, neurons, k + 1).astype(np.int64)
    rows = edges[:-1] + (rng.random((neurons, k)) * (edges[1:] - edges[:-1])).astype(np.int64)
    keep = rng.random((neurons, k)) >= 0.1
    col_ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    return col_ptr, rows[keep].astype(np.int32), rng.uniform(0.02, 0.2, (neurons, k))[keep].astype(np.float32)


class _Network:
    """The layers of a case as ``SpDNN.set_network`` takes them."""

    def __init__(self, kind, neurons, layers):
        self.kind, self.neurons = kind, neurons
        self.source = None if kind == "general" else SyntheticNetwork(neurons, layers, kind)
        self.bias = GENERAL_BIAS if kind == "general" else float(self.source.bias)

    def pattern_id(self, layer):
        return layer if self.source is None else self.source.pattern_id(layer)

    def layer_csc(self, layer):
        key = (self.kind, self.neurons, self.pattern_id(layer))
        if key not in _LAYERS:
            if len(_LAYERS) > 400:
                _LAYERS.clear()
            _LAYERS[key] = _general_layer(self.neurons, layer) if self.source is None else self.source.layer_csc(layer)
        return _LAYERS[key]


# ---- the images ----------------------------------------------------------------------------------------------------

def _blobs(neurons, batch, seed):
    """The images of ``generator.synthetic_images``, drawn on the GPU."""
    g = int(math.isqrt(neurons))
    r_mean = g * math.sqrt(0.15 * 1.17 / (math.pi * 3))
    ids = np.arange(batch, dtype=np.uint64)
    axis = torch.arange(g, device="cuda", dtype=torch.float32)
    out = torch.empty((batch, neurons), device="cuda", dtype=torch.float32)
    discs = []
    for d in range(3):
        key = ids * np.uint64(16) + np.uint64(d * 3)
        cx, cy = ((rand_unit(seed, 7, key + np.uint64(i)) * g).astype(np.float32) for i in (0, 1))
        rr = ((0.55 + 0.9 * rand_unit(seed, 7, key + np.uint64(2))) * r_mean).astype(np.float32)
        discs.append([torch.from_numpy(a).cuda()[:, None, None] for a in (cx, cy, rr)])
    step = max(1, 2 ** 26 // neurons)
    for s in range(0, batch, step):
        e = min(batch, s + step)
        on = torch.zeros((e - s, g, g), device="cuda", dtype=torch.bool)
        for cx, cy, rr in discs:
            on |= (axis[None, None, :] - cx[s:e]) ** 2 + (axis[None, :, None] - cy[s:e]) ** 2 <= rr[s:e] ** 2
        out[s:e] = on.reshape(e - s, neurons)
    return out


def _images(case, seed):
    neurons, batch = case["neurons"], case["batch"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["images"] == "mixed":
        density = 0.05 + 0.55 * torch.rand((batch, 1), device="cuda", generator=gen)
        return (torch.rand((batch, neurons), device="cuda", generator=gen) < density).float()
    y0 = _blobs(neurons, batch, seed)
    if case["images"] == "grey":
        y0 *= 0.5 + 1.5 * torch.rand((batch, neurons), device="cuda", generator=gen)
    return y0


def _packed(y0):
    """Bit matrix of a binary input: bit (n & 7) of byte n >> 3 of a row = neuron n (neurons is a multiple of 32)."""
    batch, neurons = y0.shape
    out = torch.empty((batch, neurons // 8), device="cuda", dtype=torch.uint8)
    weight = 2 ** torch.arange(8, device="cuda", dtype=torch.int32)
    step = max(1, 2 ** 26 // neurons)
    for s in range(0, batch, step):
        e = min(batch, s + step)
        out[s:e] = ((y0[s:e].view(e - s, neurons // 8, 8) != 0) * weight).sum(dim=2).to(torch.uint8)
    return out


def prepare(case, seed):
    net = _Network(case["net"], case["neurons"], case["layers"])
    engines = []
    for _ in range(2 if case["slices"] > 1 else 1):
        engine = SpDNN(case["neurons"], case["layers"], net.bias)
        engine.set_network(net)
        engines.append(engine)
    y0 = _images(case, seed)
    form = case["input"]
    if form == "coo_host":
        at = y0.nonzero().to(torch.int32).cpu().numpy()
        data = (np.ascontiguousarray(at[:, 0]) + 1, np.ascontiguousarray(at[:, 1]) + 1)
    elif form == "dense_host":
        data = y0.cpu().numpy()
    elif form == "bits_host":
        data = _packed(y0).cpu().pin_memory()
    elif form == "bits_device":
        data = _packed(y0)
    else:
        data = y0
    # result buffers the program keeps: the list of survivors has room for every image (-1 behind the last), and so have
    # the activations
    ids = np.full(case["batch"], -1, dtype=np.int32)
    rows = torch.zeros((case["batch"], case["neurons"])).pin_memory() if case["fetch"] == "all" else None
    return {"engines": engines, "data": data, "form": form, "batch": case["batch"], "slices": case["slices"], "ids": ids, "rows": rows}


def _activations(engine, rows):
    """``spdnn_get_activations`` of the C ABI into a caller's buffer (``SpDNN.activations`` allocates one per call)."""
    rc = engine._lib.spdnn_get_activations(engine._ctx, ctypes.c_void_p(rows.data_ptr()), rows.shape[0])
    if rc != 0:
        raise RuntimeError(f"spdnn_get_activations: {rc}")


def _set_input(engine, state, lo, hi):
    if state["form"] == "coo_host":
        engine.set_input_coo(state["data"][0], state["data"][1], None, state["batch"])
    elif state["form"].startswith("bits"):
        engine.set_input_bits(state["data"][lo:hi], lo)
    else:
        engine.set_input_dense(state["data"][lo:hi], lo)


def run(state):
    batch, slices, ids, rows = state["batch"], state["slices"], state["ids"], state["rows"]
    if slices == 1:
        engine = state["engines"][0]
        _set_input(engine, state, 0, batch)
        engine.infer()
        count = len(engine.categories(out=ids))
        out = {"count": count, "categories": ids, "live": engine.layer_live()}
        if rows is not None:
            _activations(engine, rows)
            out["activations"] = rows
        return out
    count, live = 0, 0
    per = -(-batch // slices)
    for i in range(slices + 1):
        if i < slices:
            e = state["engines"][i % 2]
            _set_input(e, state, i * per, min(batch, (i + 1) * per))
            e.infer_async()
        if i > 0:
            e = state["engines"][(i - 1) % 2]
            e.sync()
            count += len(e.categories(out=ids[(i - 1) * per:min(batch, i * per)]))
            live = live + e.layer_live()
    return {"count": count, "categories": ids, "live": live}


def work(case):
    """Bytes: the input once, every distinct layer's entries once, the survivors' numbers.  Flops: one multiply and add
    per entry of ONE layer and image -- how many layers an image lives, and so how much more there is to do, is decided by
    the data."""
    neurons, batch = case["neurons"], case["batch"]
    per_image = {"dense_device": 4 * neurons, "dense_host": 4 * neurons, "bits_device": neurons / 8, "bits_host": neurons / 8,
                 "coo_host": 8 * 0.15 * neurons}[case["input"]]
    if case["net"] == "radix16":
        net = SyntheticNetwork(neurons, case["layers"])
        distinct = net.num_patterns()
    else:
        distinct = case["layers"]
    entries = (28.5 * 0.9 if case["net"] == "general" else 32) * neurons
    layer = entries * (8 if case["net"] == "general" else 4)
    out = 4 * batch / 4 + (4 * neurons * batch / 4 if case["fetch"] == "all" else 0)
    return {"bytes": per_image * batch + layer * distinct + out, "flops": 2 * entries * batch}


def tolerance(case):
    # Every sum is added in ascending input order in fp32: categories, live counts and activations are the same bits.
    return "exact"
