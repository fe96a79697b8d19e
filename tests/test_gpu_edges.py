"""Edge sizes of the cluster broadphase and of the one-block path.

Broadphase (clusters of 32 segments, levels of 32 nodes): the contact lists and step limits after
a detection are bit-exact against the FP32 oracle that follows the engine's precision policy (the
same separately rounded filter decides on both sides), at segment counts on either side of a
cluster (32), of a level (1024 segments) and of the next one (32768), in batches of many tiny
scenes, and with connected vertices.

One-block path: one frame against the FP64 oracle at sizes on either side of a warp and at the
largest, in a batch of tiny scenes, and with more contacts than it holds in shared memory;
max position error / max displacement <= 1e-4, the bar of the FP32 build everywhere else, and
1e-9 x segment length in the FP64 build.  The tangle of 256 vertices runs in the FP64 build: it
amplifies rounding (two orders of summation in single precision differ by up to 2.6e-4 of the
displacement within the frame).

Newton kernels: a scene alone takes the one of its size, in a batch of its copies that of the batch's;
the states are bit for bit the same, on either side of the sizes where the kernel changes, with
connected vertices, with more contacts in a block than its helping warps take at once, and in a
settled pile, most of whose contacts are in range.
"""
import numpy as np
import pytest

import oracle
from yarnball_b200 import scenes
from yarnball_b200.sim import Sim

pytestmark = pytest.mark.gpu

H = 1.0 / 1020.0
FRAME = 1.0 / 30.0


def _walks(lens, seed, cube, glue=False, precision="fp32"):
    lens = np.asarray(lens, np.int32)
    sim = Sim(int(lens.sum()), precision=precision)
    scenes.fill_yarns(sim, scenes.random_walks_batch(seed, [len(lens)], lens, cube=cube), lens, pin_first=True)
    for k, v in scenes.PILE_META.items():
        setattr(sim.meta, k, v)
    if glue:  # the ends of every other yarn to the start of the next one, both ways
        ends = np.cumsum(lens) - 1
        for e in ends[:-1:2]:
            sim.verts["connectionIndex"][e] = e + 1
            sim.verts["connectionIndex"][e + 1] = e
    return _ready(sim)


def _ready(sim):
    sim.configure()
    sim.setKBend(1e-8)
    sim.setKStretch(2e-2)
    sim.maxH = 1e-3
    rng = np.random.default_rng(sim.numVerts)
    sim.vels[:] = rng.normal(0, 0.1, (sim.numVerts, 3))
    sim.upload()
    return sim


def _tiny_batch(count, sizes=(3, 4, 35)):
    """`count` scenes of one short wavy yarn pair each, most of less than a cluster."""
    counts = [2 * sizes[i % len(sizes)] for i in range(count)]
    sim = Sim(scenes=counts)
    off = 0
    rng = np.random.default_rng(count)
    for c in counts:
        m = c // 2
        x = np.zeros((2, m, 3), np.float32)
        x[:, :, 0] = np.arange(m) * 2e-3
        x[1, :, 1] = 0.9e-3
        x += rng.normal(0, 0.1e-3, x.shape).astype(np.float32)
        scenes.fill_yarns(sim, x.reshape(-1, 3), np.array([m, m]), offset=off, pin_first=True)
        off += c
    sim.set_meta_all(**scenes.PILE_META)
    return _ready(sim)


def _lens(segments):
    """Yarns whose segment counts sum to `segments`."""
    out, left = [], segments
    while left > 0:
        s = min(left, 97)
        if 0 < left - s < 2:
            s -= 2
        out.append(s + 1)
        left -= s
    return out


CUBE = {31: 0.008, 32: 0.008, 33: 0.008, 65: 0.01, 1023: 0.02, 1024: 0.02, 1025: 0.02, 1057: 0.02, 32767: 0.055,
        32768: 0.055, 32769: 0.055}

DETECT = {("segments %d" % s): (lambda s=s: _walks(_lens(s), s, CUBE[s])) for s in CUBE}
DETECT["connected"] = lambda: _walks(_lens(900), 5, 0.015, glue=True)
DETECT["tiny scenes"] = lambda: _tiny_batch(70)


@pytest.mark.parametrize("name", list(DETECT))
def test_cluster_pairs_find_every_contact(name):
    sim = DETECT[name]()
    orc = oracle.from_sim(sim, mode=oracle.FP32_MIXED)
    total = 0
    for mask in (1 | 2, 4):  # predictor and a rebuilt order, then the same boxes refitted
        sim.debug_phases(mask, H if mask & 1 else 0.0)
        if mask & 1:
            orc.phases(1 | 2, H)
        nc_g, lists_g, sl_g = sim.debug_contacts()
        nc_o, lists_o, sl_o = orc.contacts()
        assert np.array_equal(nc_g, nc_o)
        for i in np.nonzero(nc_g)[0]:
            assert np.array_equal(lists_g[i], lists_o[i]), i
        segs = (sim.verts["flags"] & 2) != 0
        assert np.array_equal(sl_g[segs], sl_o[segs].astype(np.float32))
        total += int(nc_g.sum())
    assert total > 0
    sim.close()
    orc.close()


SMALL = {
    "3": lambda: _walks([3], 1, 0.01),
    "31": lambda: _walks([16, 15], 2, 0.006),
    "32": lambda: _walks([16, 16], 2, 0.006),
    "33": lambda: _walks([16, 17], 2, 0.006),
    "255": lambda: _walks([51] * 5, 3, 0.012),
    "256 fp64": lambda: _walks([32] * 8, 4, 0.012, precision="fp64"),
    "256 dense": lambda: _walks([32] * 8, 6, 0.0075),
    "tiny scenes": lambda: _tiny_batch(18, (3, 4, 11)),
    "connected": lambda: _walks([20] * 10, 7, 0.012, glue=True),
}


@pytest.mark.parametrize("name", list(SMALL))
def test_one_block_sizes_vs_fp64_oracle(name):
    sim = SMALL[name]()
    assert sim.numVerts <= 256
    x0 = sim.read_state_f64()[0]
    orc = oracle.from_sim(sim, mode=oracle.FP64)
    l0 = sim.launch_count()
    sim.advance(FRAME)
    assert sim.launch_count() - l0 == 1
    orc.advance(FRAME, float(np.float32(sim.maxH)))
    pos, ref = sim.read_state_f64()[0], orc.state()["pos"]
    disp = np.abs(ref - x0).max()
    bar = 1e-9 * 2e-3 if sim.precision == "fp64" else 1e-4 * disp
    assert disp > 0 and np.abs(pos - ref).max() <= bar
    if name == "256 dense":
        assert sim.debug_contacts()[0].sum() > 2560
    sim.close()
    orc.close()


ALONE = {
    # name: (yarn lengths, cube, glue, precision)
    "257": ([128, 129], 0.02, False, "fp32"),
    "1949_glued": ([31] * 62 + [27], 0.02, True, "fp32"),
    "dense": ([125] * 16, 0.015, False, "fp32"),
    "8880": ([80] * 111, 0.04, False, "fp32"),
    "8881": ([83] * 107, 0.04, False, "fp32"),
    "257_fp64": ([128, 129], 0.02, False, "fp64"),
    "4440_fp64": ([40] * 111, 0.03, True, "fp64"),
    "4441_fp64": ([4441 // 3] * 2 + [4441 - 2 * (4441 // 3)], 0.03, False, "fp64"),
}


@pytest.mark.parametrize("name", list(ALONE))
def test_newton_kernels_of_all_sizes_agree_bit_for_bit(name):
    lens, cube, glue, precision = ALONE[name]
    sim = _walks(lens, 11, cube, glue, precision)
    copies = 30000 // sim.numVerts + 1  # past the sizes of the small blocks
    batch = Sim.gather([(sim, 0)] * copies)
    for s in (sim, batch):
        s.advance(4 * H)
    a, b = sim.read_state_f64(), batch.read_state_f64()
    for x, y in zip(a, b):
        for c in (0, copies - 1):
            o = batch.sceneOffsets[c]
            assert np.array_equal(x, y[o:o + sim.numVerts])


def test_newton_kernels_agree_bit_for_bit_in_a_settled_pile():
    sim = _walks([125] * 16, 12, 0.0197)
    for _ in range(2):
        sim.advance(FRAME)
    copies = 70  # 140,000 vertices
    batch = Sim.gather([(sim, 0)] * copies)
    for _ in range(3):  # the choice follows the contacts of the advance before
        for s in (sim, batch):
            s.advance(4 * H)
    a, b = sim.read_state_f64(), batch.read_state_f64()
    for x, y in zip(a, b):
        for c in (0, copies - 1):
            o = batch.sceneOffsets[c]
            assert np.array_equal(x, y[o:o + sim.numVerts])
