"""The work that users of this library have it do, as timed cases.

Every case runs through the public entry points:

  chain   a clip resident in device memory: Basic then Final over the whole
          clip (Session.set_clip_device, Session.render_clip_device), or both
          stages overlapped (render_chain_device)
  server  a frame server: Session.render_frame_window from several threads,
          host frames in, host frames out, `count` new frames of a long clip
          per pass
  stacks  vnlb.Basic / vnlb.Aggregate / vnlb.Final / vnlb.Aggregate on host
          arrays, the whole call
  mlp     the learned proposals' network: gradients of one batch (forward and
          backward) and the logits of one batch

Parameter sets (`preset`):

  plugin  vnlbcu's own defaults: block 7 (planes 3) or 10 (planes 1), step 3 or
          5, groups of 16 grown to 64, a 27 x 27 window, patch_time 2, rank 15
  core    the CPU core's defaults: block 8, step 8, groups of 8 grown to 32, a
          19 x 19 window, patch_time 1, rank 8
  dense   block 8, step 4, groups of 16 grown to 64 by tau 400, a 19 x 19
          window, patch_time 2, radius 2, rank 16
  mixed   block 8, step 8, groups of the rank's size grown four times by tau
          200, a 19 x 19 window, patch_time 2, rank 24 / 16 / 8 by noise level

Clips are generated on the GPU from the seed: sinusoids, a gradient and
rectangles under global motion, plus Gaussian noise of `sigma` (8-bit scale).
"""
from __future__ import annotations

import math
import random
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "vapoursynth-vnlb_b200"))

import vnlb  # noqa: E402
import vnlbcu  # noqa: E402
import vnlbgpu_lib as lib  # noqa: E402

LONG_CLIP = 1 << 20  # frames of the frame server's clip; nothing is sized by it


# --------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    clip = lambda name, w, h, n, planes, sigma, preset, form="plain", radius=1, overlap=False: dict(
        name=name, kind="chain", width=w, height=h, frames=n, planes=planes, sigma=float(sigma), preset=preset,
        form=form, radius=radius, overlap=overlap)
    return [
        # the smallest call: a thumbnail-sized gray clip, latency and launches
        clip("gray_thumb_plugin", 160, 120, 3, 1, 10, "plugin"),
        # vnlbcu.Basic / Final as users call them, on SD-like colour and HD gray
        clip("yuv_540p_plugin", 960, 540, 3, 3, 10, "plugin"),
        clip("gray_1080p_plugin", 1920, 1080, 2, 1, 15, "plugin"),
        # the same defaults with tensor-core matching
        clip("yuv_540p_plugin_tc", 960, 540, 3, 3, 10, "plugin", "chosen_tc"),
        # HD colour with the CPU core's defaults: exact, and tensor-core
        clip("yuv_1080p_core", 1920, 1080, 8, 3, 20, "core"),
        clip("yuv_1080p_core_tc", 1920, 1080, 8, 3, 20, "core", "chosen_tc"),
        # odd sizes (rows not 16-byte aligned), a wider temporal window, stages overlapped
        clip("yuv_odd_core_chain", 853, 479, 5, 3, 5, "core", "plain", 2, True),
        # dense grids and large groups, exact
        clip("gray_720p_dense", 1280, 720, 4, 1, 25, "dense", "plain", 2),
        # the largest frames, tensor-core
        clip("gray_2160p_mixed_tc", 3840, 2160, 3, 1, 15, "mixed", "chosen_tc"),
        # the plugin's getFrame path: host frames, four frame threads
        dict(name="server_720p_core", kind="server", width=1280, height=720, count=4, planes=3, sigma=20.0,
             preset="core", form="plain", radius=1, threads=4),
        # contribution stacks on host arrays with uncoupled planes
        dict(name="stacks_cif_uncoupled", kind="stacks", width=352, height=288, frames=3, planes=3, sigma=20.0,
             preset="core", form="plain", radius=1),
        # training the learned proposals (33 x 33 x 5 offsets): forward and backward of one batch
        dict(name="mlp_batch_2048", kind="mlp", batch=2048, inputs=45, hidden=128, layers=3, outputs=5445),
    ]


def draw(rng: random.Random) -> dict:
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choices(("chain", "server", "stacks", "mlp"), (12, 2, 1, 1))[0]
    if kind == "mlp":
        return dict(kind="mlp", batch=log(64, 2048), inputs=rng.choice((27, 45, 81, 135)), hidden=128, layers=3,
                    outputs=log(1083, 5445))
    preset = "core" if kind in ("server", "stacks") else rng.choice(("plugin", "core", "dense", "mixed"))
    planes = rng.choice((1, 3)) if preset in ("plugin", "core") else 1
    # the most pixels of a frame at this cost per pixel
    most = {("plugin", 3): 960 * 540, ("plugin", 1): 1920 * 1080, ("dense", 1): 1280 * 720,
            ("mixed", 1): 3840 * 2160}.get((preset, planes), 1920 * 1080)
    if kind != "chain":
        most = 1280 * 720 if kind == "server" else 352 * 288
    pixels = log(96 * 72, most)
    aspect = rng.uniform(0.75, 2.0)
    width = max(64, min(int(math.sqrt(pixels * aspect)), most // 64))
    height = max(64, pixels // width)
    if width * height > most:
        height = most // width
    case = dict(kind=kind, width=width, height=height, planes=planes,
                sigma=round(math.exp(rng.uniform(math.log(3.0), math.log(40.0))), 2), preset=preset,
                form=rng.choice(("plain", "plain", "chosen", "chosen_tc")) if kind == "chain" else "plain",
                radius=2 if preset == "dense" else (rng.choice((1, 1, 2)) if preset == "core" else 1))
    if kind == "server":
        case.update(count=rng.choice((1, 2, 4)), threads=rng.choice((1, 2, 4)))
    else:
        case.update(frames=rng.choice((2, 3)) if kind == "stacks" or preset != "core" else rng.randint(2, 8))
    if kind == "chain":
        case.update(overlap=rng.random() < 0.3)
    return case


def arguments(case: dict) -> dict:
    """The keyword arguments of both stages."""
    radius = case["radius"]
    if case["preset"] == "plugin":
        return dict(radius=radius)
    if case["preset"] == "dense":
        return dict(block_size=8, block_step=4, group_size=16, bm_range=9, radius=radius, patch_time=2, rank=16,
                    cap_factor=4.0, tau=400.0)
    if case["preset"] == "mixed":
        rank = 24 if case["sigma"] < 10 else 16 if case["sigma"] < 22 else 8
        return dict(block_size=8, block_step=8, group_size=rank, bm_range=9, radius=radius, patch_time=2, rank=rank,
                    cap_factor=4.0, tau=200.0)
    return dict(block_size=8, block_step=8, group_size=8, bm_range=9, radius=radius, patch_time=1, rank=8,
                cap_factor=4.0, variance_threshold=1.1)


def stage_parameters(case: dict, stage: int, frames: int) -> lib.Params:
    kw = arguments(case)
    if case["preset"] == "core" and stage == lib.STAGE_FINAL:
        kw.update(variance_threshold=1.7)
    if case.get("threads"):
        kw.update(num_streams=case["threads"])
    shape = np.lib.stride_tricks.as_strided(np.zeros(1, np.float32),
                                            (frames, case["planes"], case["height"], case["width"]), (0, 0, 0, 0))
    return vnlbcu.parse_parameters(stage, shape, case["sigma"], dict(kw, form=case["form"]))


# --------------------------------------------------------------------------- inputs
def make_clip(case: dict, frames: int, seed: int) -> torch.Tensor:
    """Noisy clip [frames][planes][H][W], float32 on the GPU, from the seed alone."""
    rng = random.Random(seed)
    gen = torch.Generator("cuda").manual_seed(seed)
    h, w, planes = case["height"], case["width"], case["planes"]
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    moves, x, y = [(0, 0)], 0, 0
    for _ in range(frames - 1):
        x, y = x + rng.randint(-2, 2), y + rng.randint(-2, 2)
        moves.append((x, y))
    out = torch.empty((frames, planes, h, w), device="cuda")
    for c in range(planes):
        waves = [(rng.uniform(0, math.pi), 2 * math.pi / rng.uniform(4, 64), rng.uniform(0.05, 0.15),
                  rng.uniform(0, 2 * math.pi)) for _ in range(6)]
        grad = rng.uniform(-0.15, 0.15), rng.uniform(-0.15, 0.15)
        rects = [(rng.random(), rng.random(), rng.uniform(0.05, 0.25), rng.uniform(0.05, 0.25), rng.uniform(0.1, 0.9))
                 for _ in range(10)]
        for f, (ox, oy) in enumerate(moves):
            u, v = xs + ox, ys + oy
            value = grad[0] * (u / w - 0.5) + grad[1] * (v / h - 0.5)
            for theta, k, amp, phase in waves:
                value = value + amp * torch.sin(k * (math.cos(theta) * u + math.sin(theta) * v) + phase)
            for x0, y0, rw, rh, level in rects:
                inside = (u >= x0 * w) & (u < (x0 + rw) * w) & (v >= y0 * h) & (v < (y0 + rh) * h)
                value = torch.where(inside, torch.full_like(value, level - 0.5), value)
            out[f, c] = (0.5 + (0.3 if c else 1.0) * value).clamp(0, 1)
    return out.add_(torch.randn(out.shape, device="cuda", generator=gen), alpha=case["sigma"] / 255.0)


def mlp_inputs(case: dict, seed: int):
    gen = torch.Generator("cuda").manual_seed(seed)
    x = torch.randn((case["batch"], case["inputs"]), device="cuda", generator=gen) * 0.5
    targets = torch.randint(0, case["outputs"], (case["batch"], 8), device="cuda", generator=gen, dtype=torch.int32)
    return x, targets


def server_frame(clip, n: int):
    """Frame n of the frame server's clip: the generated frames played back and forth."""
    m = n % (2 * len(clip) - 2)
    return clip[m if m < len(clip) else 2 * len(clip) - 2 - m]


SERVER_FRAMES = 8  # generated frames of the frame server's clip


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "mlp":
        x, targets = mlp_inputs(case, seed)
        net = lib.MLP(case["inputs"], case["hidden"], case["layers"], case["outputs"], max_batch=case["batch"],
                      seed=seed & 0x7FFFFFFF)
        return dict(case=case, net=net, x=x, targets=targets,
                    logits=torch.empty((case["batch"], case["outputs"]), device="cuda"))
    planes, h, w = case["planes"], case["height"], case["width"]
    if kind == "stacks":
        return dict(case=case, clip=make_clip(case, case["frames"], seed).cpu().numpy())
    frames = LONG_CLIP if kind == "server" else case["frames"]
    sessions = [lib.Session(stage_parameters(case, stage, frames), w, h, frames, planes)
                for stage in (lib.STAGE_BASIC, lib.STAGE_FINAL)]
    if kind == "server":
        clip = make_clip(case, SERVER_FRAMES, seed).cpu().numpy()
        return dict(case=case, clip=clip, basic=sessions[0], final=sessions[1], next=0, frames={},
                    pool=ThreadPoolExecutor(case["threads"]))
    clip = make_clip(case, frames, seed)
    stream = torch.cuda.Stream()
    for s in sessions:
        s.set_stream(stream.cuda_stream)
    return dict(case=case, clip=clip, basic=sessions[0], final=sessions[1], stream=stream,
                basic_out=torch.empty_like(clip), final_out=torch.empty_like(clip))


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "mlp":
        grads, loss = state["net"].gradients(state["x"].data_ptr(), state["targets"].data_ptr(), case["batch"], 8)
        state["net"].logits(state["x"].data_ptr(), case["batch"], state["logits"].data_ptr())
        return dict(gradients=grads, loss=loss, logits=state["logits"])
    if kind == "stacks":
        clip, sigma, kw = state["clip"], case["sigma"], dict(arguments(case), chroma=0)
        agg = dict(patch_time=1, radius=case["radius"])
        stacks = vnlb.Basic(clip, sigma=sigma, **kw)
        basic = vnlb.Aggregate(stacks, src=clip, **agg)
        final = vnlb.Aggregate(vnlb.Final(clip, ref=basic, sigma=sigma, **kw), src=clip, **agg)
        return dict(basic=basic, final=final, stacks=stacks)
    basic, final = state["basic"], state["final"]
    if kind == "server":
        return serve(state)
    clip, b_out, f_out = state["clip"], state["basic_out"], state["final_out"]
    basic.set_clip_device(lib.SOURCE_CLIP, clip.data_ptr(), clip)
    final.set_clip_device(lib.SOURCE_CLIP, clip.data_ptr(), clip)
    final.set_clip_device(lib.SOURCE_REF, b_out.data_ptr(), b_out)
    if case["overlap"]:
        lib.render_chain_device(basic, final, b_out.data_ptr(), f_out.data_ptr())
    else:
        basic.render_clip_device(b_out.data_ptr())
        final.render_clip_device(f_out.data_ptr())
    return dict(basic=b_out, final=f_out)


def serve(state: dict):
    """The next `count` Final frames, and the Basic frames they need that are not there yet."""
    case, clip, ready = state["case"], state["clip"], state["frames"]
    first, count = state["next"], case["count"]
    state["next"] = first + count
    ranges = [state["final"].required_source_range(n) for n in range(first, first + count)]
    need = range(min(r[0] for r in ranges), max(r[1] for r in ranges) + 1)
    for n in [n for n in ready if n < need[0]]:
        del ready[n]

    def basic_frame(n):
        lo, hi = state["basic"].required_source_range(n)
        return n, state["basic"].render_frame_window(n, [server_frame(clip, i) for i in range(lo, hi + 1)], first=lo)

    def final_frame(n):
        lo, hi = state["final"].required_source_range(n)
        return state["final"].render_frame_window(n, [server_frame(clip, i) for i in range(lo, hi + 1)],
                                                  [ready[i] for i in range(lo, hi + 1)], first=lo)

    made = [n for n in need if n not in ready]
    ready.update(state["pool"].map(basic_frame, made))
    finals = list(state["pool"].map(final_frame, range(first, first + count)))
    return dict(basic=[ready[n] for n in made], final=finals)


# --------------------------------------------------------------------------- the least work
def work(case: dict) -> dict:
    """Bytes: each input read once, each output written once.  Flops: the
    distances of every candidate (3 per sample), and per group the model (mean,
    Gram, basis) and two projections and one reconstruction of its rows, the
    groups taken as half of the grid with group_size rows each."""
    if case["kind"] == "mlp":
        h, n = case["hidden"], case["batch"]
        weights = case["inputs"] * h + (case["layers"] - 1) * h * h + h * case["outputs"]
        return dict(bytes=4.0 * (n * (case["inputs"] + 8) + 2 * weights + n * case["outputs"]),
                    flops=2.0 * 4 * n * weights)
    frames = case.get("frames", case.get("count"))
    planes, h, w = case["planes"], case["height"], case["width"]
    values = planes * h * w
    p = stage_parameters(case, lib.STAGE_BASIC, max(frames, 3))
    P, Pt = p.patch_size, p.patch_time
    grid = ((w - P) // p.proc_step + 1) * ((h - P) // p.proc_step + 1)
    window = min(p.search_window, w - P + 1) * min(p.search_window, h - P + 1)
    temporal = min(p.search_bwd + p.search_fwd + 1, max(1, frames - Pt + 1)) if case["kind"] != "server" else \
        p.search_bwd + p.search_fwd + 1
    anchors = frames - Pt + 1 if case["kind"] != "server" else frames
    dim = P * P * Pt * planes
    match = sum(3.0 * grid * window * temporal * P * P * Pt * c for c in (1, planes))
    model = 2.0 * p.similar * p.similar * dim / 2 + 2.0 * p.rank * p.similar * dim
    rows = 2.0 * 3 * p.similar * p.rank * dim
    stacks = 0
    if case["kind"] == "stacks":  # stacks written and read once, both stages
        stacks = 2 * 2 * 2.0 * frames * values * (2 * case["radius"] + 1) * 4
    return dict(bytes=4.0 * frames * values * 5 + stacks,
                flops=anchors * (match + 2 * (grid / 2) * (model + rows)))


# --------------------------------------------------------------------------- the same in 64 bits
def exact(case: dict, seed: int):
    """What run() returns, from its definition in float64: the network's
    gradients and logits with BF16-rounded weights, or the two stages of the
    filter."""
    if case["kind"] == "mlp":
        return exact_mlp(case, seed)
    total = LONG_CLIP if case["kind"] == "server" else case["frames"]
    basic_p, final_p = (stage_parameters(case, s, total) for s in (lib.STAGE_BASIC, lib.STAGE_FINAL))
    if case["kind"] == "server":
        # Final frame n reads the Basic frames up to n + 2 radius, and they the clip up to 2 radius further
        basic_n = case["count"] + 2 * case["radius"]
        frames = make_clip(case, SERVER_FRAMES, seed).double()
        clip = torch.stack([server_frame(frames, n) for n in range(basic_n + 2 * case["radius"])])
        basic, _ = exact_stage(basic_p, clip, None, total, basic_n, True)
        final, _ = exact_stage(final_p, clip[:basic_n], basic, total, case["count"], True)
        return dict(basic=list(basic), final=list(final))
    coupled = case["kind"] != "stacks"  # the stacks case filters each plane on its own
    clip = make_clip(case, total, seed).double()
    basic, stacks = exact_stage(basic_p, clip, None, total, total, coupled)
    final, _ = exact_stage(final_p, clip, basic, total, total, coupled)
    return dict(basic=basic, final=final) if coupled else dict(basic=basic, final=final, stacks=torch.stack(stacks))


def spatial_low(center: torch.Tensor, axis: int, P: int, window: int) -> torch.Tensor:
    """First patch origin of each window: centred, shifted into the frame."""
    half, top = (window - 1) // 2, axis - P
    shift = (center - half).clamp(max=0) + (center + half - top).clamp(min=0)
    return (center - half - shift).clamp(min=0)


def anchor_grid(p, anchor: int, total: int, H: int, W: int) -> torch.Tensor:
    """The staggered grid [G][2] (y, x) in raster order."""
    P, step = p.patch_size, p.proc_step
    key = (0 if anchor == total - p.patch_time else anchor) % step
    out = []
    xs = np.arange(W - P + 1)
    for y in range(H - P + 1):
        if y in (0, H - P) or y % step == key:
            phase = 0 if y == H - P else key + y // step
            keep = xs[(xs == 0) | (xs == W - P) | (xs % step == phase % step)]
            out.append(np.stack([np.full_like(keep, y), keep], 1))
    return torch.from_numpy(np.concatenate(out)).cuda()


def patch_rows(video: torch.Tensor, f: int, Pt: int, P: int, channels: int) -> torch.Tensor:
    """Every patch of frames f .. f + Pt - 1, [origins][channels * Pt * P * P]."""
    v = video[f:f + Pt, :channels].unfold(2, P, 1).unfold(3, P, 1)
    return v.permute(2, 3, 1, 0, 4, 5).reshape(v.shape[2] * v.shape[3], -1)


def exact_stage(p, clip, ref, total, out_frames, coupled):
    """One stage over the frames of `clip` (the first of `total`): the output
    frames 0 .. out_frames - 1 and every anchor frame's contribution stack."""
    F, C, H, W = clip.shape
    P, Pt, K = p.patch_size, p.patch_time, p.similar
    sb, sf, slots = p.search_bwd, p.search_fwd, p.search_bwd + p.search_fwd + p.patch_time
    search = clip if ref is None else ref
    num = torch.zeros_like(clip)
    weight = torch.zeros((F, H, W), dtype=torch.float64, device="cuda")
    center = 0.5 * (P - 1)
    r2 = ((torch.arange(P, device="cuda", dtype=torch.float64) - center) / max(center, 0.5)) ** 2
    window = torch.exp(-0.5 * (r2[:, None] + r2[None, :]))
    window = ((window / window.max()) ** p.weight_gamma).reshape(-1)
    stacks = []
    for a in range(min(total - Pt, out_frames - 1 + sb) + 1):
        shift = min(0, a - sb) + max(0, a + sf - (total - Pt))
        low, high = max(0, a - sb - shift), min(total - Pt, a + sf - shift)
        schedule = [a] + list(range(a + 1, high + 1)) + list(range(a - 1, low - 1, -1))
        grid = anchor_grid(p, a, total, H, W)
        rows = exact_match(p, search, a, schedule, grid, C if ref is not None else 1)
        alive = exact_paste(p, a, grid, rows, H, W)
        rows = {k: v[alive] for k, v in rows.items()}
        anum, aweight = exact_filter(p, clip, ref, rows, a, window, coupled)
        num += anum
        weight += aweight
        if not coupled:
            stack = torch.zeros((C, slots, 2, H, W), dtype=torch.float64, device="cuda")
            for s in range(slots):
                if 0 <= a - sb + s < F:
                    stack[:, s, 0], stack[:, s, 1] = anum[a - sb + s], aweight[a - sb + s]
            stacks.append(stack.reshape(C, slots * 2 * H, W))
    out = torch.where(weight[:, None] > 0, num / weight[:, None], clip)
    return out[:out_frames], stacks


def exact_match(p, search, a, schedule, grid, channels):
    """The retained rows of every anchor, closest first: kept, frame, y, x [G][cap]."""
    H, W = search.shape[2:]
    P, Pt = p.patch_size, p.patch_time
    G, Wx, Wy = len(grid), min(p.search_window, W - P + 1), min(p.search_window, H - P + 1)
    yl, xl = spatial_low(grid[:, 0], H, P, p.search_window), spatial_low(grid[:, 1], W, P, p.search_window)
    reference = patch_rows(search, a, Pt, P, channels)[grid[:, 0] * (W - P + 1) + grid[:, 1]]
    d = torch.empty((G, len(schedule) * Wx * Wy), dtype=torch.float64, device="cuda")
    for k, f in enumerate(schedule):
        patches = patch_rows(search, f, Pt, P, channels)
        for cell in range(Wx * Wy):
            at = (yl + cell // Wx) * (W - P + 1) + xl + cell % Wx
            d[:, k * Wx * Wy + cell] = (patches[at] - reference).square_().sum(1)
        del patches
    n = d.shape[1]
    cap = min(n, max(p.similar, math.ceil(p.similar * p.similar_cap_factor)))
    parts = [torch.sort(x, dim=1, stable=True) for x in d.split(8192)]
    dist = torch.cat([x.values[:, :cap] for x in parts])
    pick = torch.cat([x.indices[:, :cap] for x in parts])
    limit = dist[:, min(p.similar, n) - 1].clamp(min=p.tau)
    k, cell = pick // (Wx * Wy), pick % (Wx * Wy)
    return dict(kept=dist <= limit[:, None], frame=torch.tensor(schedule, device="cuda")[k],
                y=yl[:, None] + cell // Wx, x=xl[:, None] + cell % Wx)


def exact_paste(p, a, grid, rows, H, W):
    """The anchors that are processed: in raster order, each one's matches in
    the anchor frame take later anchors (at or beside them) out."""
    P, G = p.patch_size, len(grid)
    index = torch.full((H * W,), -1, dtype=torch.int64, device="cuda")
    index[grid[:, 0] * W + grid[:, 1]] = torch.arange(G, device="cuda")
    own, edges = torch.arange(G, device="cuda")[:, None].expand_as(rows["x"]), []
    here = rows["kept"] & (rows["frame"] == a)
    for dy, dx in ((0, 0), (-1, 0), (1, 0), (0, -1), (0, 1)):
        y, x = rows["y"] + dy, rows["x"] + dx
        ok = here & (y >= 0) & (y < H) & (x >= 0) & (x < W)
        ok &= {(0, 0): rows["y"] >= 0, (-1, 0): rows["y"] > 2 * P, (1, 0): rows["y"] < H - 2 * P,
               (0, -1): rows["x"] > 2 * P, (0, 1): rows["x"] < W - 2 * P}[dy, dx]
        hit = index[(y * W + x)[ok]]
        g = own[ok]
        edges.append(torch.stack([g, hit])[:, hit > g])
    edges = torch.cat(edges, 1).cpu().numpy()
    edges = edges[:, np.argsort(edges[0], kind="stable")]
    alive = bytearray(b"\1" * G)
    for g, j in zip(edges[0].tolist(), edges[1].tolist()):
        if alive[g]:
            alive[j] = 0
    return torch.from_numpy(np.frombuffer(bytes(alive), np.uint8).astype(bool)).cuda()


def exact_filter(p, clip, ref, rows, a, window, coupled):
    """The weighted filtered rows of the processed groups, summed per pixel."""
    F, C, H, W = clip.shape
    P, Pt, R = p.patch_size, p.patch_time, p.rank
    num = torch.zeros_like(clip)
    weight = torch.zeros((F, H, W), dtype=torch.float64, device="cuda")
    c, t, y, x = (i.reshape(-1).cuda() for i in torch.meshgrid(*(torch.arange(n) for n in (C, Pt, P, P)),
                                                               indexing="ij"))
    column = ((t * C + c) * H + y) * W + x
    pixel = (t * H * W + y * W + x)[:Pt * P * P]
    sigma2 = p.beta * p.sigma ** 2
    noise2 = sigma2 if ref is None else p.beta * p.sigma_basic ** 2
    member2 = max((p.sigma if ref is None else p.sigma_basic) ** 2, p.membership_noise_floor * p.sigma ** 2)
    models = [slice(0, len(column))] if coupled or C == 1 else [slice(i * Pt * P * P, (i + 1) * Pt * P * P)
                                                               for i in range(C)]
    chunk = max(64, int(4e8 / 8 / rows["x"].shape[1] / len(column)))
    for i in range(0, len(rows["x"]), chunk):
        part = {k: v[i:i + chunk] for k, v in rows.items()}
        kept = part["kept"]
        base = (part["frame"] * C * H + part["y"]) * W + part["x"]
        noisy = clip.reshape(-1)[base[:, :, None] + column]
        model = noisy if ref is None else ref.reshape(-1)[base[:, :, None] + column]
        S = kept.sum(1)
        B = S.clamp(max=p.similar)  # model rows: the closest ones
        first = (torch.arange(kept.shape[1], device="cuda")[None, :] < B[:, None]).double()
        log_weight, filtered = 0.0, torch.empty_like(noisy)
        flat = torch.zeros(len(S), dtype=torch.bool, device="cuda")
        if ref is not None and p.flat_areas:
            planes = noisy.reshape(len(S), -1, C, Pt * P * P) * kept[:, :, None, None]
            n = (S * Pt * P * P).double()[:, None]
            variance = (planes.square().sum((1, 3)) - planes.sum((1, 3)).square() / n) / (n - 1)
            flat = variance.mean(1) < p.gamma * p.sigma ** 2
        for cols in models:
            u, v = model[:, :, cols], noisy[:, :, cols]
            D = u.shape[2]
            mean = (u * first[:, :, None]).sum(1) / B[:, None]
            middle = mean
            if ref is not None:
                middle = torch.where(flat[:, None], mean, (v * first[:, :, None]).sum(1) / B[:, None])
            u, v = u - mean[:, None], v - middle[:, None]
            X = (u * first[:, :, None])[:, :p.similar]
            lam, vec = torch.linalg.eigh(X @ X.transpose(1, 2) / B[:, None, None])
            lam, vec = lam.flip(1)[:, :R], vec.flip(2)[:, :, :R]
            basis = X.transpose(1, 2) @ vec  # [n][D][R]
            length = basis.norm(dim=1, keepdim=True)
            basis = torch.where(length > 1e-9, basis / length.clamp(min=1e-300), torch.zeros_like(basis))
            signal = (lam - noise2).clamp(min=0)
            left = lam - lam.clamp(max=noise2) if noise2 > 0 else lam
            shrink = torch.where(left > p.variance_threshold * sigma2, left / (left + sigma2), torch.zeros_like(left))
            volume = torch.log1p(signal / member2).sum(1) / D
            precision = p.weight_epsilon + D / B + (signal / (signal + sigma2)).sum(1)
            projected = u @ basis
            square = projected.square()
            score = (square / (signal + member2)[:, None]).sum(2) + \
                (u.square().sum(2) - square.sum(2)).clamp(min=0) / member2
            score = (score - D) / math.sqrt(2 * D)
            least = torch.where(kept, score, torch.full_like(score, math.inf)).amin(1, keepdim=True)
            log_weight = log_weight + (-p.weight_alpha * torch.log(precision)[:, None]
                                       - p.weight_beta * (score - least + volume[:, None])) / len(models)
            filtered[:, :, cols] = middle[:, None] + ((v @ basis) * shrink[:, None]) @ basis.transpose(1, 2)
        w = torch.exp(log_weight.clamp(-80, 80)) * kept
        layer = part["frame"][:, :, None] + torch.arange(Pt, device="cuda")
        slot = layer - a + p.search_bwd
        w = w[:, :, None] * ((slot >= 0) & (slot < p.search_bwd + p.search_fwd + Pt))
        w = (w[:, :, :, None] * window).reshape(len(S), -1, Pt * P * P)
        filtered *= w.repeat(1, 1, C)
        num.view(-1).index_add_(0, (base[:, :, None] + column).reshape(-1), filtered.reshape(-1))
        base = (part["frame"] * H + part["y"]) * W + part["x"]
        weight.view(-1).index_add_(0, (base[:, :, None] + pixel).reshape(-1), w.reshape(-1))
    return num, weight


def exact_mlp(case: dict, seed: int):
    """The network with its weights rounded to BF16 and everything else in float64."""
    x, targets = mlp_inputs(case, seed)
    net = lib.MLP(case["inputs"], case["hidden"], case["layers"], case["outputs"], max_batch=1,
                  seed=seed & 0x7FFFFFFF)
    flat = torch.from_numpy(net.get_weights()).cuda()
    sizes = [case["inputs"]] + [case["hidden"]] * case["layers"] + [case["outputs"]]
    params, at = [], 0
    for fan_in, fan_out in zip(sizes, sizes[1:]):
        w = flat[at:at + fan_in * fan_out].view(fan_out, fan_in).bfloat16().double().requires_grad_()
        at += fan_in * fan_out
        b = flat[at:at + fan_out].double().requires_grad_()
        at += fan_out
        params += [w, b]
    z = x.double()
    for i in range(0, len(params), 2):
        z = z @ params[i].T + params[i + 1]
        z = torch.relu(z) if i + 2 < len(params) else z
    loss = -torch.log_softmax(z, 1).gather(1, targets.long()).mean(1).mean()
    loss.backward()
    grads = torch.cat([q.grad.reshape(-1) for q in params])
    return dict(gradients=grads, loss=loss.detach(), logits=z.detach())
