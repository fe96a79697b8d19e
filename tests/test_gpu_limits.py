"""Inputs at the limits of what the engine accepts.

Unbounded boxes: a predicted displacement whose square overflows single precision gives a segment
a box without bounds and an infinite filter distance, so it is listed with every segment of its
scene that is no neighbour of it, and with nothing else: not with the vertices that start no
segment, and not with the places past a scene's last segment in a cluster of 32.  The lists of all
broadphase paths are the same.

Configured again: a simulation of the same topology gets a fresh device state with all its segments:
boxes, contacts and states are bit for bit those of one configured once.

Walks over the BVH: its memory is taken when one of them is first chosen; where it does not fit the call
says so, the mode stays, and the simulation goes on.

A scene of more than 2^20 segments, whose clusters have a third level above them: the lists of the walk over
the BVH, and the same states.

bounds(): the box of all padded segment boxes in the build's precision, rounded to the nearest float.
"""
import numpy as np
import pytest

import oracle
from tests.test_gpu_edges import _walks
from tests.test_gpu_newton import _pairs_of_yarns
from yarnball_b200 import scenes
from yarnball_b200.sim import Sim

pytestmark = pytest.mark.gpu

H = 1e-3


def _straight_yarns(counts, fast):
    """Scenes of parallel yarns (`counts`: their lengths, scene by scene), far apart but for one
    crossing pair; vertex `fast` of each scene moves by 1e20 in a substep."""
    sizes = [sum(c) for c in counts]
    sim = Sim(scenes=sizes)
    off = 0
    for lens in counts:
        m = sum(lens)
        x = np.zeros((m, 3), np.float32)
        at = 0
        for y, length in enumerate(lens):
            x[at:at + length, 0] = np.arange(length) * 2e-3
            x[at:at + length, 1] = (0.9e-3 if y == 1 else 0.02 * y)
            at += length
        scenes.fill_yarns(sim, x, np.asarray(lens, np.int32), offset=off, pin_first=True)
        off += m
    sim.set_meta_all(**scenes.PILE_META)
    sim.configure()
    sim.maxH = H
    for o in sim.sceneOffsets[:-1]:
        sim.vels[o + fast] = (1e23, -1e23, 1e23)
    sim.upload()
    return sim


def _lists(sim):
    nc, lists, _ = sim.debug_contacts()
    return nc, lists


UNBOUNDED = {
    "one scene": [[13, 7]],
    "a cluster and a part": [[20, 20]],
    "two scenes": [[15, 6], [21, 9, 3]],
    "whole warps": [[16, 16]],
}


@pytest.mark.parametrize("name", list(UNBOUNDED))
@pytest.mark.parametrize("fast", [0, 4])
def test_unbounded_boxes_meet_segments_only(name, fast):
    counts = UNBOUNDED[name]
    got = []
    for mode in ("walk", "packets", "clusters", "one block"):
        sim = _straight_yarns(counts, fast)
        if mode == "one block":
            sim.advance(H)  # one substep; the lists are those of its detection
        else:
            sim.set_small_path(False)
            sim.set_traversal({"walk": 0, "packets": 1, "clusters": 2}[mode])
            sim.debug_phases(1 | 2, H)
        got.append(_lists(sim))
        offs, segs = sim.sceneOffsets, (sim.verts["flags"] & 2) != 0
        sim.close()
    nc, lists = got[0]
    for s in range(len(counts)):
        here = np.nonzero(segs[offs[s]:offs[s + 1]])[0] + offs[s]
        for k in range(offs[s] + max(fast - 1, 0), offs[s] + fast + 1):  # the segments at the fast vertex
            assert np.array_equal(lists[k], here[np.abs(here - k) > 2])
    for nc_x, lists_x in got[1:]:
        assert np.array_equal(nc, nc_x)
        for a, b in zip(lists, lists_x):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("small_path", [True, False])
def test_configured_again(small_path):
    def fresh():
        sim = _straight_yarns([[60, 60, 20]], 4)
        sim.vels[:] = 0
        sim.vels[:60, 1] = 0.3  # the first yarn towards the second
        return sim

    once, again = fresh(), fresh()
    for s in (once, again):
        s.set_small_path(small_path)
    again.configure()
    once.upload()
    again.upload()
    for s in (once, again):
        s.setKBend(1e-8)
        s.setKStretch(2e-2)
    # configure() scales masses and rest rotors of the present ones: give both the same
    for name in ("verts", "qs", "qRests"):
        getattr(again, name)[...] = getattr(once, name)
    for s in (once, again):
        s.upload()
    assert np.isfinite(np.concatenate(again.bounds())).all()  # before any detection
    for s in (once, again):
        s.advance(8 * H)
    assert _lists(once)[0].sum() > 0
    assert np.array_equal(_lists(once)[0], _lists(again)[0])
    assert np.array_equal(np.concatenate(once.bounds()), np.concatenate(again.bounds()))
    for a, b in zip(once.read_state_f64(), again.read_state_f64()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("small_path", [True, False])
def test_opposite_contact_forces_cancel_before_the_own_terms(small_path):
    """A yarn between two others that cross it at the same place: their forces on it are opposite and 10^5
    times its weight.  Contacts are summed first, so they cancel exactly and the weight keeps its bits; with
    the weight first, some 0.3 % of it would be rounded away.  One substep of one iteration against the
    FP64 oracle; what is left is some twenty roundings of 6e-8, the bar is 1e-5."""
    sim = Sim(18)
    line = (np.arange(6) - 2.5) * 2e-3
    x = np.zeros((3, 6, 3), np.float32)
    x[0, :, 1], x[0, :, 2] = line, 0.5e-3
    x[1, :, 0] = line
    x[2, :, 1], x[2, :, 2] = line, -0.5e-3
    scenes.fill_yarns(sim, x.reshape(-1, 3), np.array([6, 6, 6], np.int32), pin_first=False)
    sim.verts["invMass"][:6] = 0
    sim.verts["invMass"][12:] = 0
    for k, v in dict(scenes.PILE_META, kCollision=1e-2, numItr=1).items():
        setattr(sim.meta, k, v)
    sim.meta.gravity = (0.0, 0.0, -9.8)
    sim.configure()
    sim.setKBend(1e-8)
    sim.setKStretch(2e-2)
    sim.maxH = H
    sim.upload()
    sim.set_small_path(small_path)
    orc = oracle.from_sim(sim, mode=oracle.FP64)
    sim.advance(H)
    orc.advance(H, float(np.float32(H)))
    got, ref = sim.read_state_f64()[0][8, 2], orc.state()["pos"][8, 2]
    assert ref < -1e-12 and abs(got - ref) <= 1e-5 * abs(ref)
    assert {2, 14} <= set(_lists(sim)[1][8].tolist())
    sim.close()
    orc.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("traversal", [0, 2])
def test_bounds_are_the_nearest_floats(precision, traversal):
    R = np.float32 if precision == "fp32" else np.float64
    for seed in range(6):
        sim = _walks([60, 60, 37], seed, 0.02, precision=precision)
        sim.set_small_path(False)
        sim.set_traversal(traversal)
        sim.debug_phases(1 | 2, H)
        x, dx = sim.read_state_f64()[0].astype(R), sim.debug_dx().astype(R)
        reach = np.sqrt(((dx * dx)[:, 0] + (dx * dx)[:, 1]) + (dx * dx)[:, 2])
        reach = np.maximum(reach[:-1], reach[1:])
        m = sim.meta
        pad = (R(m.radius) + R(0.5) * R(m.barrierThickness)) * R(m.detectionScaler) + reach
        seg = (sim.verts["flags"][:-1] & 2) != 0
        lo = (np.minimum(x[:-1], x[1:]) - pad[:, None])[seg].min(0)
        hi = (np.maximum(x[:-1], x[1:]) + pad[:, None])[seg].max(0)
        got = sim.bounds()
        assert np.array_equal(got[0], lo.astype(np.float32)) and np.array_equal(got[1], hi.astype(np.float32))
        sim.close()


def test_bvh_memory_is_taken_with_the_first_walk():
    import torch

    from yarnball_b200._abi import YarnBallError

    n = 200000
    sims = []
    for _ in range(2):
        sim = _walks([250] * (n // 250), 3, 0.12)
        sims.append(sim)
        plain = sim.device_bytes()
        assert plain < 2000 * n
    sims[0].set_traversal(0)
    assert sims[0].device_bytes() >= plain + 250 * n
    sims[0].set_traversal(1)  # no second one
    assert sims[0].device_bytes() < plain + 260 * n
    sims[0].advance(2 * H)
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (32 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(YarnBallError):
        sims[1].set_traversal(0)
    del held
    torch.cuda.empty_cache()
    assert sims[1].device_bytes() == plain
    sims[1].advance(2 * H)
    for a, b in zip(sims[0].read_state_f64(), sims[1].read_state_f64()):
        assert np.array_equal(a, b)
    sims[1].set_traversal(0)
    for s in sims:
        s.set_traversal(2)
        s.advance(H)
        s.set_traversal(0)
        s.advance(H)
    for a, b in zip(sims[0].read_state_f64(), sims[1].read_state_f64()):
        assert np.array_equal(a, b)
    for s in sims:
        s.close()


def test_clusters_of_more_than_a_million_segments():
    states, lists = [], []
    for mode in (0, 2):
        sim = _pairs_of_yarns(2110, 250)
        assert ((sim.verts["flags"] & 2) != 0).sum() > 1 << 20
        sim.set_traversal(mode)
        for mask in (1 | 2, 4):  # a rebuilt order, then the same refitted
            sim.debug_phases(mask, H if mask & 1 else 0.0)
            lists.append(sim.debug_packed_contacts())
        sim.advance(2 * H)
        lists.append(sim.debug_packed_contacts())
        states.append(sim.read_state_f64() + sim.bounds())
        sim.close()
    for (off, cols), (off2, cols2) in zip(lists[:3], lists[3:]):
        assert off[-1] > 1 << 20
        assert np.array_equal(off, off2) and np.array_equal(cols, cols2)
    for a, b in zip(*states):
        assert np.array_equal(a, b)
