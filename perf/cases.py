"""The detector's and the JPEG decoder's performance cases.

Each case is a dict of plain values; `prepare` makes what a program holds
before the call (frames or files from a seed, a detector, server or decoder
with its families and options), `run` is one pass through the package's
public calls. Frames are the synthetic scenes of apriltags_fast_b200.synth
(no public data set exists for the benchmark): gradient, noise, tags at
random poses, filled distractor shapes.

`where` says where frames lie when the call begins: "host" (ordinary
memory, as a camera library hands them over), "pinned" (page-locked), or
"device" (already on the GPU). `scene`: "plain" (some tags on a calm
background), "dense" (24 tags per 2 megapixels and 200 shapes: many quad
candidates), "ramp" (large frames: two megapixels' worth of both, uneven
light, per-frame blur).
"""
import dataclasses
import math

import numpy as np
import torch

import apriltags_fast_b200 as AT
from apriltags_fast_b200 import synth


def _frames(name, width, height, count=1, where="host", scene="plain", families="tag36h11", bits=2, decimate=2.0,
            sigma=0.0, deglitch=False, mix="", call="detect"):
    return dict(name=name, call=call, width=width, height=height, count=count, where=where, scene=scene,
                families=families, bits=bits, decimate=decimate, sigma=sigma, deglitch=deglitch, mix=mix)


def _files(name, width, height, count, color, quality, restart, to):
    return dict(name=name, call="jpeg", width=width, height=height, count=count, color=color, quality=quality,
                restart=restart, to=to)


def listed():
    return [
        # the smallest call: one webcam frame per call, where launches and
        # waits count (a robot's control loop)
        _frames("vga_host", 640, 480),
        # an odd-sized crop (region of interest), two families
        _frames("roi_odd_host", 1279, 717, families="tag36h11,tag25h9"),
        # the drop-in form: one 1080p frame of a busy scene per call
        _frames("fhd_host", 1920, 1080, scene="dense"),
        # a few cameras' frames per call, already on the GPU
        _frames("hd_batch8_device", 1280, 720, 8, "device", call="batch"),
        # the throughput form: many busy 1080p frames on the GPU
        _frames("fhd_batch32_device", 1920, 1080, 32, "device", "dense", call="batch"),
        # the same from page-locked capture buffers
        _frames("fhd_batch32_pinned", 1920, 1080, 32, "pinned", "dense", call="batch"),
        # a mixed batch: VGA to 4K frames, each with its own family set
        _frames("mixed_batch16_device", 3840, 2160, 16, "device", families="tag36h11,tag25h9", mix="even",
                call="batch"),
        # a still camera's large frame at full resolution, a large-table
        # family beside a small one
        _frames("still_12mp_full", 4032, 3024, 1, "device", "ramp", "tagStandard52h13,tag36h11", decimate=1.0),
        # the quad image filtered, other decimation, other tag layouts
        _frames("options_batch4_host", 1280, 720, 4, "host", "dense", "tagStandard41h12,tagCircle21h7", 1, 1.5, 0.8,
                True, call="batch"),
        # frames of many streams through the request server
        _frames("served_mix32", 3840, 2160, 32, "host", mix="served", call="serve"),
        # a batch of gray camera JPEGs into device frames for the detector
        _files("jpeg_gray_batch32", 1920, 1080, 32, "gray", 90, 0, "device"),
        # one colour photo (4:2:0) into a host frame
        _files("jpeg_420_single", 1920, 1080, 1, "420", 85, 0, "host"),
    ]


_FAMILIES = ("tag36h11", "tag25h9", "tag36h11,tag25h9", "tagStandard41h12", "tag16h5", "tagStandard52h13,tag36h11")


def draw(rng):
    """One more case of the same ranges: VGA to 12 megapixel frames, 1 to 32
    a call, odd sizes among them; or JPEG files of such sizes."""
    budget = 32 * 1920 * 1080  # pixels a call at decimate 2, at most
    if rng.random() < 0.25:
        width = round(math.exp(rng.uniform(math.log(320), math.log(4032))))
        height = round(width * rng.choice((0.5625, 0.75)))
        color = rng.choice(("gray", "gray", "444", "420"))
        most = max(1, min(32, budget // (width * height) // (1 if color == "gray" else 4)))
        count = round(math.exp(rng.uniform(0, math.log(most)))) if most > 1 else 1
        case = _files("", width, height, count, color, rng.randrange(60, 96), rng.choice((0, 0, 8, 60)),
                      rng.choice(("device", "host")))
    else:
        width = round(math.exp(rng.uniform(math.log(480), math.log(4032))))
        height = round(width * rng.choice((0.5625, 0.75)))
        decimate = rng.choice((2.0, 2.0, 2.0, 2.0, 1.0, 1.5, 3.0))
        per = width * height * (4 / decimate ** 2 if decimate < 2 else 1)
        most = max(1, min(32, int(budget / per)))
        count = round(math.exp(rng.uniform(0, math.log(most)))) if most > 1 and rng.random() < 0.6 else 1
        case = _frames("", width, height, count, rng.choice(("host", "device", "pinned")),
                       rng.choice(("plain", "dense")), rng.choice(_FAMILIES), rng.choice((1, 2)), decimate,
                       rng.choice((0.0, 0.0, 0.0, 0.8, -0.6)), rng.random() < 0.15,
                       call="batch" if count > 1 else "detect")
    del case["name"]
    return case


_SCENES = {
    "plain": dict(tags=(4, 30), side=(60, 140), tilt=40.0, noise=3.0, blur=(0.7, 0.7), shapes=0, ramp=None),
    "dense": dict(tags=(24, 24), side=(30, 220), tilt=60.0, noise=4.0, blur=(0.8, 0.8), shapes=200, ramp=None),
    "ramp": dict(tags=(80, 80), side=(16, 400), tilt=65.0, noise=6.0, blur=(0.5, 1.5), shapes=1000, ramp=(0.4, 1.0)),
}


def _scene(case, width, height, families, seed):
    s = _SCENES[case.get("scene", "dense")]
    part = 1.0 if case.get("scene") == "ramp" else min(1.0, width * height / (1920 * 1080))
    tags = tuple(math.ceil(n * part) for n in s["tags"])
    side = (s["side"][0], min(s["side"][1], height // 3))
    cfg = synth.Config(width, height, families=tuple(families), ntags=tags, side=side, tilt_deg=s["tilt"],
                       noise=s["noise"], blur=s["blur"], distractors=math.ceil(s["shapes"] * part), ramp=s["ramp"])
    return synth.make_frame(cfg, seed)[0]


def _sizes(case):
    """(width, height) of each frame of the call."""
    n = case["count"]
    if case.get("mix") == "even":
        return [((640, 480), (1280, 720), (1920, 1080), (3840, 2160))[i % 4] for i in range(n)]
    if case.get("mix") == "served":  # of ten frames: six 720p, three 1080p, one 4K
        order = (0, 1, 0, 0, 1, 0, 2, 0, 1, 0)
        return [((1280, 720), (1920, 1080), (3840, 2160))[order[i % 10]] for i in range(n)]
    return [(case["width"], case["height"])] * n


def _pictures(case, seed):
    """The call's frames, all different: scenes drawn new for a part of them
    (at most 8 of a size, 1 of 4K), the others the same scenes turned half
    round or with the camera moved."""
    families = case.get("families", "tag36h11").split(",")
    rng = np.random.default_rng(seed)
    made, out = {}, []
    for i, (w, h) in enumerate(_sizes(case)):
        fam = [families[(i // 4) % len(families)]] if case.get("mix") == "even" else families
        pool, used = made.setdefault((w, h, tuple(fam)), ([], [0]))
        most = 8 if w * h <= 2100000 and not case.get("mix") else 1
        if len(pool) < most:
            pool.append(_scene(case, w, h, fam, int(rng.integers(1 << 31))))
            out.append(pool[-1])
            continue
        k = used[0]
        used[0] += 1
        img = pool[k % len(pool)]
        turn, move = (k // len(pool)) % 2 == 0, k // len(pool) // 2
        img = img[::-1, ::-1] if turn else img
        shift = (17 * move + 8 * (not turn), 29 * move)
        out.append(np.ascontiguousarray(np.roll(img, shift, (0, 1))))
    return out, families


def _place(img, where):
    if where == "device":
        return torch.from_numpy(np.array(img)).cuda()
    if where == "pinned":
        return torch.from_numpy(np.array(img)).pin_memory().numpy()
    return img


def prepare(case, seed):
    if case["call"] == "jpeg":
        pictures, _ = _pictures(case, seed)
        sampling = (2, 2) if case["color"] == "420" else (1, 1)
        files = []
        for img in pictures:
            if case["color"] != "gray":  # the scene under coloured light
                g = img.astype(np.int16)
                img = np.stack([g, np.clip(g + 20 - (g >> 2), 0, 255), 255 - (g >> 1)], -1).astype(np.uint8)
            files.append(synth.encode_jpeg(img, case["quality"], sampling, case["restart"]))
        return {"call": "jpeg", "to": case["to"], "files": files, "decoder": AT.JpegDecoder()}
    pictures, families = _pictures(case, seed)
    det = AT.Detector(families, case["bits"], quad_decimate=case["decimate"], quad_sigma=case["sigma"],
                      deglitch=case["deglitch"])
    state = {"call": case["call"], "detector": det, "frames": [_place(p, case["where"]) for p in pictures], "masks": None,
             "found": np.zeros(_ROOM * case["count"], AT.DETECTION_DTYPE), "counts": np.zeros((2, case["count"]), np.int64)}
    if case["mix"] == "even":
        state["masks"] = [1 << ((i // 4) % len(families)) for i in range(case["count"])]
    if case["call"] == "serve":
        state["server"] = AT.Server(det, workers=2, max_batch=8)
    return state


_ROOM = 128  # detections a frame that the program's result table has room for


def _keep(state, frames, nquads):
    """All detections of the call into the program's table, one frame's
    after the other's (the rest of the table empty), with each frame's
    detection and quad counts."""
    table, counts, at = state["found"], state["counts"], 0
    for i, rec in enumerate(frames):
        table[at:at + len(rec)] = rec
        at += len(rec)
        counts[0, i], counts[1, i] = len(rec), nquads[i]
    table[at:] = 0
    return {"counts": counts, **{k: table[k] for k in AT.DETECTION_DTYPE.names}}


def run(state):
    if state["call"] == "jpeg":
        dec = state["decoder"]
        frames, errors = (dec.decode_device if state["to"] == "device" else dec.decode)(state["files"])
        return {"frames": frames, "errors": np.array(errors, np.int32)}
    det, frames = state["detector"], state["frames"]
    if state["call"] == "detect":
        found = det.detect(frames[0])
        rec = np.array([dataclasses.astuple(d) for d in found], AT.DETECTION_DTYPE)
        return _keep(state, [rec], [det.nquads])
    if state["call"] == "batch":
        found = det.detect_batch(frames, state["masks"], as_arrays=True)
        return _keep(state, found, det.last_batch_nquads)
    server = state["server"]
    for i, img in enumerate(frames):
        if not server.submit(img, user=i):
            raise RuntimeError("the server turned a frame away")
    done = {}
    while len(done) < len(frames):
        for r in server.poll(wait_ms=1000):
            if r["status"] != 0:
                raise RuntimeError(f"a served frame failed ({r['status']})")
            done[r["user"]] = r
    order = range(len(frames))
    return _keep(state, [done[i]["detections"] for i in order], [done[i]["nquads"] for i in order])


def work(case):
    """Each input byte read once, each result written once. Nothing here is
    a contraction; the floating point work depends on the scene and is
    small beside the passes over the pixels."""
    px = sum(w * h for w, h in _sizes(case))
    if case["call"] == "jpeg":
        # the entropy-coded bytes of these scenes: about 0.1 to 0.25 a pixel
        return {"bytes": px + int(px * 0.2), "flops": 0}
    tags = {"plain": 15, "dense": 24, "ramp": 80}[case["scene"]]
    return {"bytes": px + 168 * tags * case["count"], "flops": 0}


def exact(case, seed):
    """Nothing: decoded frames are bytes, and a detection's numbers are by
    contract the bits that the reference detector's own mix of 32 and 64 bit
    steps gives, not the rounding of an exact value."""
    return None
