"""Workloads of the inter-analysis stage and the steps around it, through the package's public entry points.

A case is one picture's work (or one step of many streams' pictures) as an encoder built on this package has it
done, or one pass of the proposer network. `kind` says which calls a pass makes:

- ``replay``   the drop-in form: the source and the newest reference pictures go in (device pointers), the
               P picture is analysed against the caller's decisions (`analyse_replay_device`);
- ``auto``     the batched form: one `InterBatch.step` for `streams` streams of uneven sizes;
- ``bpic``     the B-picture searches of one picture (`ironav_analyse_b_replay_device`);
- ``recon``    the caller decided: inter residual coding and reconstruction of a P picture
               (`ironav_code_inter_picture_device`), then the deblocking filter (`deblock_device`);
- ``decide``   one stream's whole P picture without the bitstream: reference planes, decide mode, the filter's
               records, the filter;
- ``bdecide``  the same for many streams in one `InterBatch.decide` (CAVLC or CABAC), records and
               `InterBatch.deblock`;
- ``encode``   `DeviceEncoder.encode_device` over a short group of pictures: an IDR picture and P pictures,
               bytes out;
- ``propose``  the proposer's forward pass over every macroblock of a picture;
- ``train``    one training step of the proposer (host samples, forward, backward, Adam).

Pictures are generated on the GPU from the seed, with the settings of `ironav_b200.synth`'s sequences: 4-octave
value noise panned by up to 6 samples a picture in quarter samples, textured rectangles moving at up to 12
samples a picture, Gaussian noise of sigma 3; chroma from the 2x2 luma means.
"""
import math
import random

import numpy as np
import torch

from ironav_b200.encoder import DeviceEncoder
from ironav_b200.inter import (BRESULT_DTYPE, DBK_MB_DTYPE, DBK_SLICE_DTYPE, INTERCODE_DTYPE, INTERDEC_DTYPE, KIND_INTER, MBCODE_DTYPE,
                               MBRESULT_DTYPE, MBSTATE_B_DTYPE, MBSTATE_DTYPE, InterBatch, InterStage, b_decision_states, reference_slices)
from ironav_b200.learned import picture_samples
from ironav_b200.proposer import Proposer

CORES = 8  # host cores of the encoder whose slice count is taken (reference_slices)
BATCH_SIZES = [(640, 360), (854, 480), (1280, 720), (1920, 1080)]  # the batched configuration's resolutions
NOUT, NFEAT = 13, 32 * 48 * 48
SHAPES = [("w1", (9, 32, 16)), ("b1", (32,)), ("w2", (9, 32, 32)), ("b2", (32,)), ("w3", (9, 32, 32)), ("b3", (32,)), ("w4", (9, 32, 32)),
          ("b4", (32,)), ("hw", (NOUT, NFEAT)), ("hb", (NOUT,))]
LR = 1e-3


def listed():
    return [
        # the smallest call: a CIF picture of a conferencing stream
        {"name": "replay_cif", "kind": "replay", "w": 352, "h": 288, "bd": 8, "refs": 1, "qp": 26, "fast": False, "sub8": False},
        # a size that is no multiple of 16, two references, sub-partitions of 8x8: the slow presets of an SD stream
        {"name": "replay_480p_2refs", "kind": "replay", "w": 854, "h": 480, "bd": 8, "refs": 2, "qp": 24, "fast": False, "sub8": True},
        # the benchmark's picture
        {"name": "replay_1080p", "kind": "replay", "w": 1920, "h": 1080, "bd": 8, "refs": 1, "qp": 27, "fast": False, "sub8": False},
        # a 4K picture at 10 bits, as HDR material is coded
        {"name": "replay_2160p_10bit", "kind": "replay", "w": 3840, "h": 2160, "bd": 10, "refs": 1, "qp": 27, "fast": False, "sub8": False},
        # a transcoding host: 32 streams of the batched configuration's resolutions a step
        {"name": "auto_32_streams", "kind": "auto", "streams": 32, "bd": 8, "qp": 27, "fast": False},
        # a B picture between two P pictures
        {"name": "bpic_1080p", "kind": "bpic", "w": 1920, "h": 1080, "bd": 8, "qp": 29, "fast": False},
        # an encoder that keeps its own decision on the host: coding and filtering of what it chose
        {"name": "recon_1080p", "kind": "recon", "w": 1920, "h": 1080, "bd": 8, "qp": 27},
        # live coding of one stream with CAVLC, the constrained-baseline form
        {"name": "decide_1080p", "kind": "decide", "w": 1920, "h": 1080, "bd": 8, "qp": 27, "refs": 1, "fast": False, "cabac": False},
        # 16 streams with the default encoder's CABAC decision in one launch
        {"name": "bdecide_16_cabac", "kind": "bdecide", "streams": 16, "bd": 8, "qp": 27, "fast": False, "cabac": True},
        # the whole default encoder on one stream: an IDR picture and three P pictures, High profile
        {"name": "encode_1080p_cabac", "kind": "encode", "w": 1920, "h": 1080, "bd": 8, "qp": 27, "pictures": 4, "cabac": True, "refs": 1},
        # the learned form's network on every macroblock of a picture
        {"name": "propose_1080p", "kind": "propose", "w": 1920, "h": 1080},
        # its training, at the training program's batch size
        {"name": "train_512", "kind": "train", "batch": 512},
    ]


def draw(rng):
    def size(lo, hi):  # an even width and height, spread over the logarithm of the area, 4:3 to 21:9
        area = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        ratio = rng.uniform(4 / 3, 21 / 9)
        w = max(64, int(math.sqrt(area * ratio)) // 2 * 2)
        return w, max(48, int(area / w) // 2 * 2)

    kind = rng.choice(["replay", "replay", "auto", "bpic", "recon", "decide", "bdecide", "encode", "propose", "train"])
    bd = rng.choice([8, 8, 10])
    qp = rng.randrange(20, 36)
    fast = rng.random() < 0.25
    if kind == "replay":
        w, h = size(176 * 144, 3840 * 2160 // 2)
        return {"kind": kind, "w": w, "h": h, "bd": bd, "refs": rng.choice([1, 1, 2, 3]), "qp": qp, "fast": fast, "sub8": rng.random() < 0.3}
    if kind == "auto":
        return {"kind": kind, "streams": int(math.exp(rng.uniform(0, math.log(33)))), "bd": bd, "qp": qp, "fast": fast}
    if kind == "bdecide":
        return {"kind": kind, "streams": int(math.exp(rng.uniform(0, math.log(13)))), "bd": 8, "qp": qp, "fast": fast, "cabac": rng.random() < 0.6}
    if kind == "propose":
        w, h = size(176 * 144, 1920 * 1080)
        return {"kind": kind, "w": w, "h": h}
    if kind == "train":
        return {"kind": kind, "batch": int(math.exp(rng.uniform(math.log(17), math.log(513))))}
    w, h = size(176 * 144, 1920 * 1080)
    case = {"kind": kind, "w": w, "h": h, "bd": bd, "qp": qp}
    if kind == "bpic":
        case["fast"] = fast
    elif kind == "decide":
        case |= {"refs": rng.choice([1, 1, 2]), "fast": fast, "cabac": rng.random() < 0.5}
    elif kind == "encode":
        case |= {"pictures": rng.choice([2, 3, 4]), "cabac": rng.random() < 0.6, "refs": rng.choice([1, 1, 3])}
    return case


# ---- pictures ---------------------------------------------------------------------------------------------


def _noise(g, h, w):
    """4-octave value noise (periods 64, 32, 16, 8), 16 to 235."""
    out = torch.zeros((h, w), device="cuda")
    for o in range(4):
        p = 64 >> o
        lat = torch.rand((1, 1, h // p + 2, w // p + 2), generator=g, device="cuda")
        up = torch.nn.functional.interpolate(lat, scale_factor=p, mode="bilinear", align_corners=False)
        out += up[0, 0, :h, :w] * (0.5 ** o)
    return 16 + out * (219 / 1.875)


def _frames(w, h, n, seed, bd):
    """n luma pictures (uint8, or int16 holding 10-bit samples) of one seeded sequence, on the GPU."""
    r = random.Random(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    margin = 6 * n + 2
    back = _noise(g, h + 2 * margin, w + 2 * margin)
    objects = []
    for _ in range(max(1, min(32, round(8 * w * h / (1920 * 1080))))):
        ow, oh = (min(r.randrange(64, 257), s // 2) for s in (w, h))
        objects.append((_noise(g, oh, ow), r.uniform(0, w - ow), r.uniform(0, h - oh), r.uniform(-12, 12), r.uniform(-12, 12)))
    qx = qy = 4 * margin
    out = []
    for t in range(n):
        x, fx, y, fy = qx // 4, (qx % 4) / 4, qy // 4, (qy % 4) / 4
        s = back[y:y + h + 1, x:x + w + 1]
        s = s[:, :-1] * (1 - fx) + s[:, 1:] * fx
        f = s[:-1] * (1 - fy) + s[1:] * fy
        for tex, ox, oy, vx, vy in objects:
            a, b = (int(min(max(p + t * v, 0), m - k)) for p, v, m, k in ((oy, vy, h, tex.shape[0]), (ox, vx, w, tex.shape[1])))
            f[a:a + tex.shape[0], b:b + tex.shape[1]] = tex
        f = f + 3.0 * torch.randn((h, w), generator=g, device="cuda")
        out.append((f.round().clamp(0, 255).to(torch.uint8) if bd == 8 else (4 * f).round().clamp(0, 1023).to(torch.int16)).contiguous())
        qx += r.randint(-24, 24)
        qy += r.randint(-24, 24)
    return out


def _chroma(y, bd):
    m = torch.nn.functional.avg_pool2d(y[None, None].float(), 2)[0, 0].round().int()
    half = 1 << (bd - 1)
    return torch.stack([half + (((m - half) * 3) >> 2), half - ((m - half) >> 1)]).to(y.dtype).contiguous()


def _bytes(n):
    return torch.zeros(n, dtype=torch.uint8, device="cuda")


def _upload(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


def _check(status, what):
    if status:
        raise RuntimeError("%s: status %d" % (what, status))


class _Stream:
    """One stream's context and device pictures: `refs` references (oldest first) and the picture to code."""

    def __init__(self, w, h, bd, seed, refs=1, chroma=False, cabac=False):
        self.w, self.h, self.bd = w, h, bd
        mb_h = (h + 15) // 16
        self.nslices = reference_slices(mb_h, CORES)
        self.st = InterStage(w, h, max_refs=refs, nslices=self.nslices, bd=bd)
        self.st.set_stream(torch.cuda.current_stream().cuda_stream)
        self.y = _frames(w, h, refs + 2, seed, bd)
        self.refs, self.src = self.y[1:-1], self.y[-1]
        self.c_refs = [_chroma(f, bd) for f in self.refs] if chroma else None
        self.c_src = _chroma(self.src, bd) if chroma else None
        n = self.st.nmb
        self.col, self.states = _bytes(n * MBSTATE_DTYPE.itemsize), _bytes(n * MBSTATE_DTYPE.itemsize)
        self.results = _bytes(n * MBRESULT_DTYPE.itemsize)
        if chroma:
            self.st.set_entropy(cabac, True)
            self.codes, self.mbs = _bytes(n * MBCODE_DTYPE.itemsize), _bytes(n * DBK_MB_DTYPE.itemsize)
            self.rec_y = torch.zeros((self.st.mb_h * 16, self.st.mb_w * 16), dtype=self.src.dtype, device="cuda")
            self.rec_c = torch.zeros((2, self.st.mb_h * 8, self.st.mb_w * 8), dtype=self.src.dtype, device="cuda")
            self.slices = np.zeros(self.nslices, dtype=DBK_SLICE_DTYPE)

    def first_column(self, qp):
        """The newest reference's own decisions, against the picture before it (its co-located vectors)."""
        self.st.push_reference_device(self.y[0].data_ptr(), self.w, self.w, self.h, None)
        self.st.set_source_device(self.refs[-1].data_ptr(), self.w)
        self.st.begin_p_picture(self.qpp(qp))
        self.st.analyse_auto_device(self.col.data_ptr(), self.results.data_ptr())
        self.st.sync()

    def qpp(self, qp):
        return qp + 6 * (self.bd - 8)

    def load(self, chroma):
        """The references (the newest with its decisions) and the source into the context."""
        st, w, h = self.st, self.w, self.h
        st.clear_references()
        for k, f in enumerate(self.refs):
            st.push_reference_device(f.data_ptr(), w, w, h, self.col.data_ptr() if k == len(self.refs) - 1 else None)
            if chroma:
                c = self.c_refs[k]
                _check(st.lib.ironav_push_reference_chroma_device(st.ctx, c[0].data_ptr(), c[1].data_ptr(), w // 2, w // 2, h // 2), "chroma")
        self.load_source(chroma)

    def load_source(self, chroma):
        st, w = self.st, self.w
        st.set_source_device(self.src.data_ptr(), w)
        if chroma:
            _check(st.lib.ironav_set_source_chroma_device(st.ctx, self.c_src[0].data_ptr(), self.c_src[1].data_ptr(), w // 2), "chroma")

    def decide(self):
        st, y, c = self.st, self.rec_y, self.rec_c
        _check(st.lib.ironav_decide_p_picture_device(st.ctx, self.states.data_ptr(), self.codes.data_ptr(), y.data_ptr(), y.shape[1],
                                                     c[0].data_ptr(), c[1].data_ptr(), c.shape[2]), "decide")

    def records(self):
        _check(self.st.lib.ironav_decide_dbk_records_device(self.st.ctx, self.codes.data_ptr(), self.states.data_ptr(), self.mbs.data_ptr()),
               "records")

    def deblock(self):
        y, c = self.rec_y, self.rec_c
        self.st.deblock_device(y.data_ptr(), y.shape[1], c[0].data_ptr(), c[1].data_ptr(), c.shape[2], self.mbs.data_ptr(), self.slices)


def _mix(case, seed):
    """The sizes of a batch's streams: drawn once for a number of streams, so that every seed has the same work."""
    r = random.Random(case["streams"])
    return [r.choice(BATCH_SIZES) + (seed * 1000 + k,) for k in range(case["streams"])]


# ---- the proposer -----------------------------------------------------------------------------------------


def _weights(seed):
    """The network's parameters as a training run starts from them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    parts = []
    for name, shape in SHAPES:
        p = torch.randn(shape, generator=g, device="cuda")
        if name == "w1":
            p *= math.sqrt(2.0 / 18)
            p[:, :, 2:] = 0
        elif name[0] == "w":
            p *= math.sqrt(2.0 / 288)
        elif name == "hw":
            p *= 0.5 / math.sqrt(NFEAT)
        else:
            p *= 0.02
        parts.append(p.reshape(-1))
    return torch.cat(parts)


def _training_batch(case, seed):
    """Two pictures' device luma, and `batch` macroblocks of them with targets."""
    w, h = 1920, 1080
    pics = [_frames(w, h, 2, seed * 7 + k, 8) for k in range(2)]
    r = np.random.default_rng(seed)
    n = case["batch"]
    which = r.integers(0, 2, n)
    mb = r.integers(0, 120 * 68, n)
    mv = np.clip(np.round(r.normal(0, 14, (n, 2))), -128, 128).astype(np.int16)
    cls = r.choice(5, n, p=[0.6, 0.2, 0.07, 0.07, 0.06]).astype(np.uint8)
    return w, h, pics, which, mb, mv, cls


def _proposer_input(cur, ref, mbx, mby):
    """The network's input [n, 2, 48, 48] in 64 bits: the macroblock tiled 3x3 and the window around it."""
    h, w = cur.shape
    i = torch.arange(48, device="cuda")
    cy, cx = (mby[:, None] * 16 + (i & 15)).clamp(max=h - 1), (mbx[:, None] * 16 + (i & 15)).clamp(max=w - 1)
    wy, wx = (mby[:, None] * 16 - 16 + i).clamp(0, h - 1), (mbx[:, None] * 16 - 16 + i).clamp(0, w - 1)
    a = cur[cy[:, :, None], cx[:, None, :]]
    b = ref[wy[:, :, None], wx[:, None, :]]
    return torch.stack([a, b], 1).double() / 255


def _named(flat):
    out, off = {}, 0
    for name, shape in SHAPES:
        n = math.prod(shape)
        out[name] = flat[off:off + n].view(shape)
        off += n
    return out


def _network(p, x):
    """The proposer in 64 bits: 4 convolutions with ReLU and the head, the features ordered (pixel, channel)."""
    n = x.shape[0]
    for l in (1, 2, 3, 4):
        wt = p["w%d" % l][:, :, :x.shape[1]]
        pad = torch.nn.functional.pad(x, (1, 1, 1, 1))
        cols = torch.stack([pad[:, :, t // 3:t // 3 + 48, t % 3:t % 3 + 48] for t in range(9)], 1)  # [n, tap, in, 48, 48]
        y = torch.einsum("toi,ntip->nop", wt, cols.reshape(n, 9, x.shape[1], 2304)) + p["b%d" % l][None, :, None]
        x = torch.relu(y).view(n, 32, 48, 48)
    return x.reshape(n, 32, 2304).permute(0, 2, 1).reshape(n, NFEAT) @ p["hw"].T + p["hb"]


# ---- the interface ----------------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "replay":
        k = s["stream"] = _Stream(case["w"], case["h"], case["bd"], seed, case["refs"])
        k.first_column(case["qp"])
        # the decisions that the caller's own loop ends with: the stage's
        k.load(False)
        k.st.begin_p_picture(k.qpp(case["qp"]), nrefs_active=case["refs"], fast=case["fast"], sub8=case["sub8"])
        k.st.analyse_auto_device(k.states.data_ptr(), k.results.data_ptr())
        k.st.sync()
    elif kind == "auto":
        ks = s["streams"] = [_Stream(w, h, case["bd"], sd) for w, h, sd in _mix(case, seed)]
        for k in ks:
            k.first_column(case["qp"])
        s["batch"] = InterBatch([k.st for k in ks])
    elif kind == "bpic":
        k = s["stream"] = _Stream(case["w"], case["h"], case["bd"], seed, 2)
        # list 0: the older picture; list 1: the newer one, with its own decisions; the B picture lies between them
        k.refs, k.src = [k.y[0], k.y[2]], k.y[1]
        st, w, h = k.st, k.w, k.h
        st.push_reference_device(k.y[0].data_ptr(), w, w, h, None)
        st.set_source_device(k.y[2].data_ptr(), w)
        st.begin_p_picture(k.qpp(case["qp"] - 2))
        st.analyse_auto_device(k.col.data_ptr(), k.results.data_ptr())
        k.load(False)
        s["bstates"], s["bresults"] = _bytes(st.nmb * MBSTATE_B_DTYPE.itemsize), _bytes(st.nmb * BRESULT_DTYPE.itemsize)
        _analyse_b(s)
        st.sync()
        s["bstates"] = _upload(b_decision_states(s["bresults"].cpu().numpy().view(BRESULT_DTYPE)))
    elif kind == "recon":
        k = s["stream"] = _Stream(case["w"], case["h"], case["bd"], seed, 1, chroma=True)
        k.first_column(case["qp"])
        k.load(True)
        k.st.begin_p_picture(k.qpp(case["qp"]))
        k.decide()
        k.records()
        k.st.sync()
        codes = k.codes.cpu().numpy().view(MBCODE_DTYPE)
        d = np.zeros(len(codes), dtype=INTERDEC_DTYPE)
        d["mode"] = np.where(codes["kind"] != KIND_INTER, 0, np.where(codes["skip"] != 0, 1, 2))
        for f in ("part", "sub", "refs", "mvs"):
            d[f] = codes[f]
        s["decs"], s["out"] = _upload(d), _bytes(len(d) * INTERCODE_DTYPE.itemsize)
        s["intra"] = (k.rec_y.clone(), k.rec_c.clone())  # the caller's planes with its intra macroblocks
    elif kind == "decide":
        k = s["stream"] = _Stream(case["w"], case["h"], case["bd"], seed, case["refs"], chroma=True, cabac=case["cabac"])
        k.first_column(case["qp"])
    elif kind == "bdecide":
        ks = s["streams"] = [_Stream(w, h, case["bd"], sd, chroma=True, cabac=case["cabac"]) for w, h, sd in _mix(case, seed)]
        for k in ks:
            k.first_column(case["qp"])
            k.load(True)
        s["batch"] = InterBatch([k.st for k in ks])
    elif kind == "encode":
        w, h, n = case["w"], case["h"], case["pictures"]
        s["enc"] = DeviceEncoder(w, h, case["qp"], keyint=n, refs=case["refs"], nslices=reference_slices((h + 15) // 16, CORES), bd=case["bd"],
                                 cabac=case["cabac"])
        s["y"] = _frames(w, h, n, seed, case["bd"])
        s["c"] = [_chroma(f, case["bd"]) for f in s["y"]]
        s["bytes"], s["used"] = [np.zeros(s["enc"].st.nmb * 384, dtype=np.uint8) for _ in range(n)], [0] * n
    elif kind == "propose":
        w, h = case["w"], case["h"]
        s["y"] = _frames(w, h, 2, seed, 8)
        smp = picture_samples(s["y"][1].data_ptr(), s["y"][0].data_ptr(), w, h, w, w)
        s["samples"], s["n"] = _upload(smp), len(smp)
        s["prop"] = Proposer(max_batch=len(smp))
        s["prop"].load_state_dict({"params": _weights(seed).cpu().numpy(), "step": 0})
    elif kind == "train":
        w, h, s["pics"], which, mb, mv, cls = _training_batch(case, seed)
        every = np.stack([picture_samples(b.data_ptr(), a.data_ptr(), w, h, w, w) for a, b in s["pics"]])
        s["samples"] = every[which, mb]
        s["mv"], s["cls"] = torch.from_numpy(mv).cuda(), torch.from_numpy(cls).cuda()
        s["prop"] = Proposer(max_batch=case["batch"])
        s["prop"].load_state_dict({"params": _weights(seed).cpu().numpy(), "step": 0})
    return s


def _analyse_b(s):
    k, case = s["stream"], s["case"]
    st, qpp = k.st, k.qpp(case["qp"])
    _check(st.lib.ironav_begin_b_picture_device(st.ctx, qpp, st.lib.ironav_lambda(qpp), 1, 0, k.col.data_ptr(), 1, 2, int(case["fast"])), "begin b")
    _check(st.lib.ironav_analyse_b_replay_device(st.ctx, s["bstates"].data_ptr(), s["bresults"].data_ptr()), "b")


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "replay":
        k = s["stream"]
        k.load(False)
        k.st.begin_p_picture(k.qpp(case["qp"]), nrefs_active=case["refs"], fast=case["fast"], sub8=case["sub8"])
        k.st.analyse_replay_device(k.states.data_ptr(), k.results.data_ptr())
        return {"results": k.results}
    if kind == "auto":
        ks = s["streams"]
        for k in ks:
            k.st.begin_p_picture(k.qpp(case["qp"]), fast=case["fast"])
        s["batch"].step([k.src.data_ptr() for k in ks], [k.refs[-1].data_ptr() for k in ks], [k.col.data_ptr() for k in ks],
                        [k.states.data_ptr() for k in ks], [k.results.data_ptr() for k in ks])
        return {"states": [k.states for k in ks], "results": [k.results for k in ks]}
    if kind == "bpic":
        k = s["stream"]
        k.load_source(False)
        _analyse_b(s)
        return {"results": s["bresults"]}
    if kind == "recon":
        k = s["stream"]
        y, c = k.rec_y, k.rec_c
        y.copy_(s["intra"][0])
        c.copy_(s["intra"][1])
        _check(k.st.lib.ironav_code_inter_picture_device(k.st.ctx, k.qpp(case["qp"]), s["decs"].data_ptr(), s["out"].data_ptr(), y.data_ptr(),
                                                         y.shape[1], c[0].data_ptr(), c[1].data_ptr(), c.shape[2]), "code")
        k.deblock()
        return {"codes": s["out"], "y": y, "c": c}
    if kind == "decide":
        k = s["stream"]
        k.load(True)
        k.st.begin_p_picture(k.qpp(case["qp"]), nrefs_active=case["refs"], fast=case["fast"])
        k.decide()
        k.records()
        k.deblock()
        return {"states": k.states, "codes": k.codes, "y": k.rec_y, "c": k.rec_c}
    if kind == "bdecide":
        ks = s["streams"]
        for k in ks:
            k.load_source(True)
            k.st.begin_p_picture(k.qpp(case["qp"]), fast=case["fast"])
        ys, cs = [k.rec_y.data_ptr() for k in ks], [k.rec_y.shape[1] for k in ks]
        cb, cr, ct = [k.rec_c[0].data_ptr() for k in ks], [k.rec_c[1].data_ptr() for k in ks], [k.rec_c.shape[2] for k in ks]
        s["batch"].decide([k.states.data_ptr() for k in ks], [k.codes.data_ptr() for k in ks], ys, cs, cb, cr, ct)
        for k in ks:
            k.records()
        s["batch"].deblock(ys, cs, cb, cr, ct, [k.mbs.data_ptr() for k in ks], [k.slices for k in ks])
        return {"codes": [k.codes for k in ks], "y": [k.rec_y for k in ks], "c": [k.rec_c for k in ks]}
    if kind == "encode":
        w = case["w"]
        for t, buf in enumerate(s["bytes"]):  # each picture's bytes into a buffer of the raw picture's size, zeros after them
            data = s["enc"].encode_device(s["y"][t].data_ptr(), s["c"][t][0].data_ptr(), s["c"][t][1].data_ptr(), w,
                                          s["y"][t - 1].data_ptr() if t else None)
            buf[:len(data)] = np.frombuffer(data, dtype=np.uint8)
            buf[len(data):s["used"][t]] = 0
            s["used"][t] = len(data)
        return {"bytes": s["bytes"], "y": s["enc"].d_rec, "c": s["enc"].d_rec_c}
    if kind == "propose":
        p, n = s["prop"], s["n"]
        p.set_samples_device(s["samples"].data_ptr(), n)
        p.forward(n)
        return {"out": p.out[:n]}
    p = s["prop"]
    p.train_step(s["samples"], s["mv"], s["cls"], lr=LR)
    return {"out": p.out[:case["batch"]], "params": p.p, "m": p.m, "v": p.v}


def _sizes(case):
    return [(case["w"], case["h"])] if "w" in case else [x[:2] for x in _mix(case, 0)]


def work(case):
    """Bytes of one pass: each input picture and record read once, each output record and plane written once (the
    search itself is integer work on data that stays on the chip); the network's passes also count the
    convolutions' and the head's multiply-adds."""
    kind = case["kind"]
    if kind in ("propose", "train"):
        n = case["batch"] if kind == "train" else sum(((w + 15) // 16) * ((h + 15) // 16) for w, h in _sizes(case))
        layers = [2 * 9 * 2 * 32 * 2304] + 3 * [2 * 9 * 32 * 32 * 2304] + [2 * NFEAT * NOUT]
        params = sum(math.prod(s) for _, s in SHAPES)
        if kind == "propose":
            return {"bytes": n * (2 * 256 + 4 * NOUT) + 2 * params, "flops": n * sum(layers)}
        # every activation is needed twice: written by the forward pass and read by the backward pass
        return {"bytes": n * (4 * 2 * 2 * NFEAT + 4 * 2304) + 28 * params, "flops": n * (3 * sum(layers) - layers[0])}
    B = 1 if case["bd"] == 8 else 2
    total = 0
    for w, h in _sizes(case):
        n = ((w + 15) // 16) * ((h + 15) // 16)
        planes = 4 * (16 * ((w + 15) // 16) + 96) * (16 * ((h + 15) // 16) + 96) * B
        luma, frame = w * h * B, 3 * w * h * B // 2
        if kind == "replay":
            total += luma + case["refs"] * (luma + planes) + n * (72 + 104)
        elif kind == "auto":
            total += 2 * luma + planes + n * (72 + 72 + 104)
        elif kind == "bpic":
            total += 3 * luma + n * (72 + 140 + 200)
        elif kind == "recon":
            total += 3 * frame + n * (78 + 1324 + 192)
        elif kind in ("decide", "bdecide"):
            total += 3 * frame + case.get("refs", 1) * planes + n * (72 + 72 + 1516)
        else:
            total += case["pictures"] * (3 * frame + planes + n * (72 + 1516))
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    kind = case["kind"]
    if kind == "propose":
        ref, cur = _frames(case["w"], case["h"], 2, seed, 8)
        mb_w, mb_h = (case["w"] + 15) // 16, (case["h"] + 15) // 16
        p = _named(_weights(seed).double())
        i = torch.arange(mb_w * mb_h, device="cuda")
        return {"out": torch.cat([_network(p, _proposer_input(cur, ref, j % mb_w, j // mb_w)) for j in i.split(128)])}
    if kind == "train":
        w, h, pics, which, mb, mv, cls = _training_batch(case, seed)
        n = case["batch"]
        flat = _weights(seed).double().requires_grad_(True)
        which, mb = torch.from_numpy(which).cuda(), torch.from_numpy(mb).cuda()
        mv, cls = torch.from_numpy(mv).cuda().double() / 128, torch.from_numpy(cls).cuda().long()
        x = torch.empty((n, 2, 48, 48), dtype=torch.float64, device="cuda")
        for k, (a, b) in enumerate(pics):
            at = (which == k).nonzero()[:, 0]
            x[at] = _proposer_input(b, a, mb[at] % 120, mb[at] // 120)
        grad, outs = torch.zeros_like(flat), []
        for at in torch.arange(n, device="cuda").split(64):
            out = _network(_named(flat), x[at])
            dist = (out[:, :8].view(-1, 4, 2) - mv[at][:, None]).abs().sum(2)
            loss = dist.min(1).values.sum() + 0.05 * dist.sum() + torch.nn.functional.cross_entropy(out[:, 8:], cls[at], reduction="sum")
            grad += torch.autograd.grad(loss / n, flat)[0]
            outs.append(out.detach())
        m, v = 0.1 * grad, 0.001 * grad * grad
        lr = torch.full_like(grad, LR)
        lr[-(NOUT * NFEAT + NOUT):] = LR / 30
        params = flat.detach() - lr * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
        return {"out": torch.cat(outs), "params": params, "m": m, "v": v}
    return None
