"""Which Newton kernel runs, and that the choice is not observable.

A scene alone takes the kernel of its size, in a batch of its copies that of the batch's size, and
`debug_newton_kernel` names it; on either side of every size where it changes, in a large batch
whose contacts are all in range (the kernel that evaluates every contact), and however few contacts
are staged, the states are the same bit for bit.
"""
import numpy as np
import pytest

from tests.test_gpu_edges import H, _ready, _walks
from yarnball_b200 import scenes
from yarnball_b200.sim import Sim

pytestmark = pytest.mark.gpu


def _pile(n, precision="fp32", density=140e6):
    lens = [80] * (n // 80) + ([n % 80] if n % 80 >= 3 else [])
    lens[0] += n - sum(lens)
    return _walks(lens, 21, round((n / density) ** (1 / 3), 4), precision=precision)


def _same_state(sim, batch, copies):
    for x, y in zip(sim.read_state_f64(), batch.read_state_f64()):
        for c in (0, copies - 1):
            o = batch.sceneOffsets[c]
            assert np.array_equal(x, y[o:o + sim.numVerts])


SIZES = [
    # vertices, precision, kernel (148 SMs)
    (8880, "fp32", "k_iter_small"),
    (8881, "fp32", "k_iter_bal<32,256>"),
    (13320, "fp32", "k_iter_bal<32,256>"),
    (13321, "fp32", "k_iter_bal<32,128>"),
    (26640, "fp32", "k_iter_bal<32,128>"),
    (26641, "fp32", "k_iter_bal<128> plain"),
    (4440, "fp64", "k_iter_small"),
    (4441, "fp64", "k_iter_bal<32,128>"),
    (13320, "fp64", "k_iter_bal<32,128>"),
    (13321, "fp64", "k_iter_bal<128> plain"),
]


@pytest.mark.parametrize("n,precision,kernel", SIZES)
def test_kernel_of_each_size_agrees_bit_for_bit(n, precision, kernel):
    sim = _pile(n, precision)
    copies = (120000 if precision == "fp32" else 30000) // n + 1
    batch = Sim.gather([(sim, 0)] * copies)
    assert sim.debug_newton_kernel()[0] == kernel
    assert batch.debug_newton_kernel()[0] == ("k_iter_bal<128>" if precision == "fp32" else "k_iter_bal<128> plain")
    for s in (sim, batch):
        s.advance(4 * H)
    assert sim.collisionStats()[0] > n  # pairs
    _same_state(sim, batch, copies)


def _pairs_of_yarns(count, verts):
    """Pairs of parallel yarns 0.9 barrier reaches apart, the pairs far from each other: every listed
    contact is in range."""
    x = np.zeros((count, 2, verts, 3), np.float32)
    x[..., 0] = np.arange(verts) * 2e-3
    x[:, 1, :, 1] = 0.9e-3
    x[..., 2] = (np.arange(count) * 0.02)[:, None, None]
    x += np.random.default_rng(count).normal(0, 0.02e-3, x.shape).astype(np.float32)
    sim = Sim(count * 2 * verts)
    scenes.fill_yarns(sim, x.reshape(-1, 3), np.full(2 * count, verts, np.int32), pin_first=True)
    for k, v in scenes.PILE_META.items():
        setattr(sim.meta, k, v)
    return _ready(sim)


def test_kernel_that_evaluates_every_contact_agrees_bit_for_bit():
    sim = _pairs_of_yarns(8, 125)
    sim.vels[:] = 0
    sim.upload()
    copies = 70  # 140,000 vertices
    batch = Sim.gather([(sim, 0)] * copies)
    assert batch.debug_newton_kernel()[0] == "k_iter_bal<128>"
    # the choice follows the contacts of the advance before; the barrier pushes the yarns out of range
    # within some ten substeps, and contacts are tested first again
    kernels = []
    for _ in range(6):
        for s in (sim, batch):
            s.advance(4 * H)
        assert sim.debug_newton_kernel()[0] == "k_iter_small"
        kernels.append(batch.debug_newton_kernel()[0])
        _same_state(sim, batch, copies)
    assert kernels[0] == "k_iter_all" and kernels[-1] == "k_iter_bal<128>"


@pytest.mark.parametrize("n,precision", [(2000, "fp32"), (9000, "fp32"), (20000, "fp32"), (30000, "fp32"),
                                         (2000, "fp64"), (9000, "fp64"), (20000, "fp64")])
def test_staged_contacts_are_not_observable(n, precision):
    states = []
    for slots in (None, 7, 1, 0):
        sim = _pile(n, precision, density=250e6)
        if slots is not None:
            sim.debug_limit_staging(slots)
            assert sim.debug_newton_kernel()[1] == slots
        sim.advance(4 * H)
        assert sim.debug_contacts()[0].sum() > 7 * n
        states.append(sim.read_state_f64())
        sim.close()
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a, b)


def _long_crossings(count, length, seed):
    """`count` scenes of two yarns of two segments each, `length` metres long against a barrier reach of
    1 mm, crossing at a small angle with a gap close to the reach."""
    rng = np.random.default_rng(seed)
    sim = Sim(scenes=[6] * count)
    x = np.zeros((count, 2, 3, 3))
    x[:, 0, :, 0] = (np.arange(3) - 1) * length
    angle = np.exp(rng.uniform(np.log(0.01), np.log(0.2), count))
    t = (np.arange(3) - 1)[None, :] * length - rng.uniform(-0.9, 0.9, (count, 1)) * length
    x[:, 1, :, 0] = -rng.uniform(0.1, 0.9, (count, 1)) * length + t * np.cos(angle)[:, None]
    x[:, 1, :, 1] = t * np.sin(angle)[:, None]
    x[:, 1, :, 2] = rng.uniform(0.99e-3, 1.03e-3, (count, 1))
    for s in range(count):
        scenes.fill_yarns(sim, x[s].reshape(-1, 3).astype(np.float32), np.array([3, 3], np.int32), offset=6 * s,
                          pin_first=False)
    sim.set_meta_all(**dict(scenes.PILE_META, kCollision=1e-5))
    sim.configure(1e-9)
    sim.setKBend(1e-8)
    sim.setKStretch(2e-2)
    sim.maxH = 1e-3
    sim.upload()
    return sim


@pytest.mark.parametrize("length", [0.02, 2.0, 20.0, 60.0])
def test_contacts_of_long_segments_are_not_skipped(length):
    """The bound that leaves contacts out holds however long the segments are against the barrier's reach:
    the states are those of evaluating every contact (which is what happens with none staged)."""
    sims = [_long_crossings(1500, length, 5) for _ in range(2)]
    sims[1].debug_limit_staging(0)
    for s in sims:
        s.advance(H)
    assert sims[0].debug_contacts()[0].sum() > 1500
    for a, b in zip(sims[0].read_state_f64(), sims[1].read_state_f64()):
        assert np.array_equal(a, b)


def _yarns(n):
    sim = Sim(n)
    x = np.zeros((n, 3), np.float32)
    x[:, 0] = np.arange(n) % 250 * 2e-3
    x[:, 1] = np.arange(n) // 250 * 5e-3
    scenes.fill_yarns(sim, x, np.full(n // 250, 250, np.int32), pin_first=True)
    for k, v in scenes.PILE_META.items():
        setattr(sim.meta, k, v)
    return sim


def test_staged_contacts_follow_the_size_and_what_fits():
    """The number of staged contacts is a rule of the simulation's size, whatever else is on the device; where
    that many do not fit, 7 or 1 are taken, and the states are the same bit for bit."""
    import torch

    n = 1000000
    sim = _ready(_yarns(n))
    assert sim.debug_newton_kernel()[1] == 16
    sim.advance(2 * H)
    state = sim.read_state_f64()
    size = {16: sim.device_bytes()}
    sim.close()
    for slots in (7, 1):
        size[slots] = size[16] - (16 - slots) * 28 * n
    room = {16: 2 * size[16], 7: (size[7] + size[16]) // 2, 1: (size[1] + size[7]) // 2}
    for slots, free in room.items():
        torch.cuda.empty_cache()
        held = torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")
        sim = _ready(_yarns(n))
        assert sim.debug_newton_kernel()[1] == slots
        del held
        torch.cuda.empty_cache()
        sim.advance(2 * H)
        for a, b in zip(state, sim.read_state_f64()):
            assert np.array_equal(a, b)
        sim.close()
