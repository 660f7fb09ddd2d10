"""Performance cases of the superimposition path, each through the entry point a program calls.

A case is one pass over a set of seeded synthetic tracks (the generators of
``supertrack_b200.workloads``), from the tracks a program has in hand to the spectra it reads back.
``mode`` says how the program calls the library:

  noalloc   st_superimpose_noalloc on one device track (C ABI, no device allocation);
  fresh     every pass clears the queue, submits the tracks again and runs them (a program that
            meets new tracks all the time);
  resident  the tracks stay queued; every pass resets the histograms and runs the batch again
            (more oversamples of a fixed track library, a parameter study);
  plain     as resident, one track at a time (the reference's per-task loop);
  host      as resident with tracks in pinned host memory, uploaded by every pass;
  served    a burst of jobs through the continuous-batching server, one spectrum per job.

Sizes, generators and histograms are those of the benchmark configurations (4,000-deposit proton
tracks, 1e6-deposit ion tracks at 2 nm, 4e6-deposit ion tracks at 10 nm, the uneven lognormal mix)
and odd sizes around them.
"""
import ctypes as C
import math

import numpy as np
import torch

import supertrack_b200 as st
import supertrack_b200.workloads as W
from supertrack_b200 import _capi

# a 64-bit result is computed up to these sizes: (oversamples of all tracks, deposit*oversamples)
EXACT_LIMIT = (20_000, 2.0e9)


def _case(name, mode, generator, tracks, deposits, diameter, oversamples, hist, **more):
    kind, bins, lower, upper = hist
    c = {"name": name, "mode": mode, "generator": generator, "tracks": tracks,
         "deposits": deposits, "diameter": diameter, "oversamples": oversamples,
         "hist": kind, "bins": bins, "lower": lower, "upper": upper, "half_length": 2500.0,
         "core_sigma": 5.0, "pen_max": 500.0, "zshift": "none", "precision": 64, "mix": 3}
    c.update(more)
    return c


LIN3000 = ("lin", 3000, 0.01, 300.0)
LOG500 = ("log", 500, 0.1, 1e4)
LOG200 = ("log", 200, 0.01, 1e4)


def listed():
    return [
        # the smallest call there is: one short proton track, a plug-in that may not allocate
        _case("noalloc-proton-4000", "noalloc", "proton", 1, 4000, 10.0, 10, LIN3000),
        # one proton track of an odd length as it comes out of a transport code: submitted, run
        # and read at once, with z measured from the voxel's face
        _case("fresh-proton-19997", "fresh", "proton", 1, 19_997, 2.0, 100, LOG200,
              zshift="minus"),
        # one dense ion track, few oversamples: must spread over the whole GPU
        _case("fresh-ion-300007", "fresh", "ion", 1, 300_007, 10.0, 10, LIN3000),
        # the small configuration: 64 proton tracks, one shared spectrum
        _case("proton-64x4000", "resident", "proton", 64, 4000, 10.0, 10, LIN3000),
        # the same kind of tracks in the reference's one-track-at-a-time loop
        _case("plain-proton-16x4000", "plain", "proton", 16, 4000, 10.0, 10, LIN3000),
        # the batched configuration: uneven tracks of both kinds, every diameter and oversample
        # count, one spectrum per track
        _case("uneven-2048", "resident", "mixed", 2048, 20_000, 0.0, 0, LOG200),
        # the same mix with the single-precision geometry option
        _case("uneven-512-fp32", "resident", "mixed", 512, 20_000, 0.0, 0, LOG200,
              precision=32, mix=5),
        # the dense configuration: 1e6-deposit ion tracks on 2 nm spheres, nearly every hit its
        # own sphere
        _case("ion-16x1e6-2nm", "resident", "ion", 16, 1_000_000, 2.0, 100, LOG500,
              half_length=5000.0),
        # the largest tracks: 4e6 deposits, thousands of hits in a sphere
        _case("ion-8x4e6-10nm", "resident", "ion", 8, 4_000_000, 10.0, 50, LIN3000,
              half_length=5000.0, core_sigma=3.0, pen_max=1000.0),
        # uneven tracks read from files: pinned host memory, uploaded by every pass
        _case("host-uneven-256", "host", "mixed", 256, 20_000, 0.0, 0, LOG200, mix=7),
        # a burst of arriving jobs at the server
        _case("served-256", "served", "mixed", 256, 20_000, 0.0, 0, LOG200, mix=11),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    mode = rng.choice(["noalloc", "fresh", "fresh", "resident", "resident", "resident",
                       "resident", "plain", "host", "served"])
    generator = rng.choice(["proton", "ion"] if mode in ("noalloc", "fresh", "plain")
                           else ["proton", "ion", "mixed"])
    hist = rng.choice([LIN3000, LOG500, LOG200])
    diameter = rng.choice([2.0, 10.0, 100.0, 1000.0])
    oversamples = logint(1, 100)
    more = {"half_length": rng.choice([2500.0, 5000.0]),
            "zshift": rng.choice(["none", "none", "plus", "minus"]),
            "mix": rng.randrange(1, 1 << 20)}
    if mode == "noalloc":
        tracks, deposits = 1, logint(500, 16_000)
    elif mode == "fresh":
        tracks, deposits = logint(1, 8), logint(500, 1_000_000)
    elif mode == "plain":
        tracks, deposits = logint(2, 32), logint(500, 200_000)
    elif generator == "mixed":
        tracks, deposits, diameter, oversamples = logint(32, 512), 20_000, 0.0, 0
    else:
        tracks, deposits = logint(4, 512), logint(500, 1_000_000)
    if generator != "mixed":
        # at most 8e6 deposits and 2.5e8 deposit*oversamples in a drawn case
        tracks = max(1, min(tracks, 8_000_000 // deposits))
        oversamples = max(1, min(oversamples, 250_000_000 // (tracks * deposits)))
    if mode in ("resident", "fresh") and rng.random() < 0.2:
        more["precision"] = 32
    c = _case("", mode, generator, tracks, deposits, diameter, oversamples, hist, **more)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------
# tracks
# ------------------------------------------------------------------------------------------------
def _shapes(case):
    """(sizes, proton?, diameter, oversamples) of every track: the case's own, whatever the seed."""
    n = int(case["tracks"])
    if case["generator"] == "mixed":
        most = 500_000 if case["mode"] in ("served", "host") else 2_000_000
        sizes, proton, d, n_os = W.config2_sizes(n, int(case["mix"]), 1.0, most)
        return sizes, proton, d, n_os.astype(np.int64)
    return (np.full(n, int(case["deposits"]), dtype=np.int64),
            np.full(n, case["generator"] == "proton"), np.full(n, float(case["diameter"])),
            np.full(n, int(case["oversamples"]), dtype=np.int64))


def _fitted(half_length, d):
    """(N, HL', L, gSO, r) of the lattice fitted into the voxel."""
    n = math.floor(half_length * 2 / d)
    length = n * d
    hl = length / 2
    r = d / 2
    if r > hl:
        n, hl = 1, r
        length = 2 * hl
    return n, hl, length, -hl + r, r


def _tracks(case, seed):
    """The deposits of all tracks, concatenated on the GPU: [x, y, z, edep], and each track's
    first deposit. Tracks are generated a few at a time, which bounds the temporaries, and with
    torch's deterministic scans, so that a seed gives the same deposits bit for bit."""
    before = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        return _generate(case, seed)
    finally:
        torch.use_deterministic_algorithms(before)


def _generate(case, seed):
    sizes, proton, diameter, _ = _shapes(case)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed) * 1_000_003 + 17)
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64)
    out = [torch.empty(int(sizes.sum()), dtype=torch.float64, device=dev) for _ in range(4)]
    hl = float(case["half_length"])
    for kind in (True, False):
        rows = np.nonzero(proton == kind)[0]
        at = 0
        while at < len(rows):
            end, total = at, 0
            while end < len(rows) and (end == at or total + sizes[rows[end]] <= 8_000_000):
                total += int(sizes[rows[end]])
                end += 1
            part = rows[at:end]
            sz = torch.as_tensor(sizes[part], device=dev)
            made = (W.gen_proton(g, sz, dev) if kind else
                    W.gen_ion(g, sz, hl, float(case["core_sigma"]), float(case["pen_max"]), dev))
            first = 0
            for j in part:
                o, n = int(offsets[j]), int(sizes[j])
                for k in range(4):
                    out[k][o:o + n] = made[k][first:first + n]
                if case["zshift"] != "none":
                    # z as measured from the voxel's lower or upper face
                    h = _fitted(hl, float(diameter[j]))[1]
                    out[2][o:o + n] += h if case["zshift"] == "minus" else -h
                first += n
            del made
            at = end
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return out, offsets


def _job_seed(seed):
    return int(seed) * 7919 + 101


# ------------------------------------------------------------------------------------------------
# what a program has in hand
# ------------------------------------------------------------------------------------------------
class _State:
    pass


def _views(case, seed, arrays, offsets):
    sizes, _, diameter, n_os = _shapes(case)
    n = len(sizes)
    views, descs = (_capi.st_track_view * n)(), (_capi.st_job_desc * n)()
    for j in range(n):
        v, d = views[j], descs[j]
        v.x, v.y, v.z, v.edep = [a.data_ptr() + 8 * int(offsets[j]) for a in arrays]
        v.n, v.on_device = int(sizes[j]), 1
        d.half_length, d.sphere_diameter = float(case["half_length"]), float(diameter[j])
        d.zshift, d.shift_track = st.ZSHIFT[case["zshift"]], 1
        d.n_oversamples, d.hist_id = int(n_os[j]), -1
        d.seed, d.track_id = _job_seed(seed), j
    return views, descs


def _submit_all(s):
    for o, n, kw in s.jobs:
        if s.host:
            s.ctx.submit(*[a[o:o + n] for a in s.arrays], **kw)
        else:
            s.ctx.submit(*[a.data_ptr() + 8 * o for a in s.arrays], on_device=True, n=n, **kw)


def prepare(case, seed):
    s = _State()
    s.mode = case["mode"]
    s.hist = (case["hist"], int(case["bins"]), float(case["lower"]), float(case["upper"]))
    s.arrays, s.offsets = _tracks(case, seed)
    sizes, _, diameter, n_os = _shapes(case)
    bins = s.hist[1]
    if s.mode == "noalloc":
        views, descs = _views(case, seed, s.arrays, s.offsets)
        s.view, s.desc, s.stats = views[0], descs[0], _capi.st_job_stats()
        s.kind = st.HIST_TYPES[s.hist[0]]
        s.counts = torch.zeros(bins, dtype=torch.int64, device="cuda")
        s.yfy = torch.zeros(bins, dtype=torch.float64, device="cuda")
        return s
    if s.mode == "served":
        s.views, s.descs = _views(case, seed, s.arrays, s.offsets)
        n = len(sizes)
        s.arrival = np.zeros(n, dtype=np.int64)
        s.counts, s.yfy = np.zeros((n, bins), dtype=np.int64), np.zeros((n, bins))
        s.server = st.Server(0, budget_bytes=32_000_000_000,
                             max_track_deposits=int(sizes.max()), max_batch_jobs=1024)
        return s
    s.host = s.mode == "host"
    if s.host:
        s.arrays = [a.cpu().pin_memory() for a in s.arrays]
        torch.cuda.empty_cache()
    s.ctx = st.Context(0)
    if int(case["precision"]) == 32:
        s.ctx.set_param("precision", 32)
    # a track has its own spectrum in the uneven mix, one spectrum sums all tracks otherwise
    own = case["generator"] == "mixed"
    ids = [s.ctx.histogram(*s.hist) for _ in range(len(sizes) if own else 1)]
    s.jobs = [(int(s.offsets[j]), int(sizes[j]),
               dict(half_length=float(case["half_length"]), sphere_diameter=float(diameter[j]),
                    n_oversamples=int(n_os[j]), hist=ids[j if own else 0],
                    seed=_job_seed(seed), track_id=j, zshift=case["zshift"]))
              for j in range(len(sizes))]
    total = s.ctx.total_bins()
    s.counts = torch.zeros(total, dtype=torch.int64).pin_memory()
    s.yfy = torch.zeros(total, dtype=torch.float64).pin_memory()
    s.read_stats = len(sizes) <= 64  # a program of many tracks reads its spectra only
    if s.mode != "fresh":
        _submit_all(s)
    return s


def run(state):
    s = state
    if s.mode == "noalloc":
        s.counts.zero_()
        s.yfy.zero_()
        kind, bins, lower, upper = s.hist
        rc = _capi.lib().st_superimpose_noalloc(C.byref(s.view), C.byref(s.desc), s.kind, bins,
                                                lower, upper, s.counts.data_ptr(),
                                                s.yfy.data_ptr(), None, C.byref(s.stats))
        _capi.check(rc, "st_superimpose_noalloc")
        return {"counts": s.counts, "yfy": s.yfy,
                "stats": np.array([s.stats.hits, s.stats.spheres, s.stats.binned,
                                   s.stats.inbox], dtype=np.int64)}
    if s.mode == "served":
        s.server.replay(s.views, s.descs, s.arrival, s.hist, s.counts, s.yfy)
        s.server.drain(60.0)
        done = s.server.poll(4096)
        return {"counts": s.counts, "yfy": s.yfy,
                "failed": int(np.count_nonzero(done["status"]))}
    ctx = s.ctx
    ctx.reset_histogram()
    if s.mode == "fresh":
        ctx.clear()
        _submit_all(s)
    else:
        ctx.jobs_reset()
    ctx.run("plain" if s.mode == "plain" else "batched")
    ctx.read_all_into(s.counts.data_ptr(), s.yfy.data_ptr(), s.counts.numel())
    out = {"counts": s.counts, "yfy": s.yfy}
    if s.read_stats:
        got = [ctx.stats(j) for j in range(len(s.jobs))]
        out["stats"] = np.array([[g["hits"], g["spheres"], g["binned"], g["inbox"]] for g in got],
                                dtype=np.int64)
    return out


def work(case):
    """Each deposit read once, each spectrum written once; the reference's FP64 operations per
    deposit and oversample (2 for the shift, 17 for lattice, distance and key) of the deposits
    that lie in the voxel's depth: a proton track is a line longer than the voxel."""
    sizes, proton, _, n_os = _shapes(case)
    spectra = len(sizes) if case["generator"] == "mixed" or case["mode"] == "served" else 1
    inside = np.where(proton, np.minimum(1.0, 2 * float(case["half_length"]) / (1.2 * sizes)), 1.0)
    return {"bytes": float(32 * sizes.sum() + 16 * int(case["bins"]) * spectra),
            "flops": float((19.0 * inside * sizes * n_os).sum())}


# ------------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ------------------------------------------------------------------------------------------------
def _philox(counter, key):
    c, (k0, k1), m = list(counter), key, 0xFFFFFFFF
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(p1 >> 32) ^ c[1] ^ k0, p1 & m, (p0 >> 32) ^ c[3] ^ k1, p0 & m]
    return c


def _shift(seed, track, os, length, hl):
    r = _philox([os, track & 0xFFFFFFFF, track >> 32, 0x53484654],
                (seed & 0xFFFFFFFF, seed >> 32))
    return [((v >> 8) + 1) * 2.0 ** -24 * length - hl for v in r[:2]]


def _edges(case):
    """Bin edges with the single-precision steps of the histogram's definition."""
    lo, hi, n = np.float32(case["lower"]), np.float32(case["upper"]), int(case["bins"])
    i = np.arange(n + 1)
    if case["hist"] == "log":
        a, b = np.float32(math.log10(float(lo))), np.float32(math.log10(float(hi)))
        return np.array([math.pow(10.0, float(a) + k * float((b - a) / np.float32(n))) for k in i])
    return float(lo) + i * float((hi - lo) / np.float32(n))


def exact(case, seed):
    sizes, _, diameter, n_os = _shapes(case)
    if n_os.sum() > EXACT_LIMIT[0] or (sizes * n_os).sum() > EXACT_LIMIT[1]:
        return None
    arrays, offsets = _tracks(case, seed)
    own = case["generator"] == "mixed" or case["mode"] == "served"
    edges = torch.as_tensor(_edges(case), device="cuda")
    bins = int(case["bins"])
    yfy = torch.zeros((len(sizes) if own else 1, bins), dtype=torch.float64, device="cuda")
    for j in range(len(sizes)):
        d = float(diameter[j])
        n, hl, length, gso, r = _fitted(float(case["half_length"]), d)
        x, y, z, e = [a[int(offsets[j]):int(offsets[j]) + int(sizes[j])] for a in arrays]
        z = z + {"plus": hl, "minus": -hl, "none": 0.0}[case["zshift"]]
        ok = z.abs() < hl
        x, y, z, v = x[ok], y[ok], z[ok], e[ok] / ((2.0 / 3.0) * d)
        a = z - gso
        kz = torch.round(a / d)
        dz2 = (kz * d - a) ** 2
        kz = kz.long() * (n * n)
        for os in range(int(n_os[j])):
            sx, sy = _shift(_job_seed(seed), j, os, length, hl)
            x1, y1 = x + sx, y + sy
            at = torch.nonzero((x1.abs() < hl) & (y1.abs() < hl)).flatten()
            ax, ay = x1[at] - gso, y1[at] - gso
            kx, ky = torch.round(ax / d), torch.round(ay / d)
            dist = ((kx * d - ax) ** 2 + (ky * d - ay) ** 2) + dz2[at]
            hit = dist <= r * r
            at = at[hit]
            key = kx[hit].long() + ky[hit].long() * n + kz[at]
            ids, inverse = torch.unique(key, return_inverse=True)
            if ids.numel() == 0:
                continue
            total = torch.zeros(ids.numel(), dtype=torch.float64, device="cuda")
            total.index_add_(0, inverse, v[at])
            b = torch.searchsorted(edges, total, right=True) - 1
            inside = (b >= 0) & (b < bins)
            yfy[j if own else 0].index_add_(0, b[inside], total[inside])
    out = yfy.cpu().numpy()
    return {"yfy": out if case["mode"] == "served" else out.reshape(-1)}
