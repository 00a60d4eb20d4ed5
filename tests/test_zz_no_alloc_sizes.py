"""pcc_soft_forces_noalloc at the sizes where its kernels change form: a lane
group's and a block's cells, the scan's tile, entry counts around eight (one
round of a group) and 32 (the ranked lists), and the largest call.  Against a
contact-by-contact numpy sum; rtol 1e-12 covers the rounding of the Hertz
power and of sums of up to a few hundred terms of one sign pattern or another
relative to the largest term."""
from __future__ import annotations

import numpy as np
import pytest

from pcc_b200 import abi
from test_zz_no_alloc import MAX_CELLS, MAX_CONTACTS, _entry

pytestmark = pytest.mark.gpu

KCC = 1333.0


def contacts(n: int, m: int, hubs: list[int], seed: int) -> dict:
    """m random contacts, then hub cells 0, 1, ... with the given entry counts more."""
    rng = np.random.default_rng(seed)
    gi, gj = rng.integers(0, n, m), rng.integers(0, n, m)
    for k, d in enumerate(hubs):
        if n > len(hubs) + 1:
            other = rng.integers(len(hubs), n, d)
            side = rng.random(d) < 0.5
            gi, gj = np.concatenate([gi, np.where(side, k, other)]), np.concatenate([gj, np.where(side, other, k)])
    o = rng.permutation(gi.size)
    c = gi.size
    nrm = rng.normal(size=(c, 3))
    return {"gid_i": gi[o].astype(np.int32), "gid_j": gj[o].astype(np.int32), "sd": rng.uniform(-0.2, 0.05, c),
            "normal": nrm / np.linalg.norm(nrm, axis=1, keepdims=True), "r_i": rng.uniform(-1, 1, (c, 3)),
            "r_j": rng.uniform(-1, 1, (c, 3)), "stress_i": rng.uniform(0, 0.5, c),
            "stress_j": rng.uniform(0, 0.5, c)}


def plain(c: dict, n: int, diameter):
    over = np.maximum(-c["sd"], 0.0)
    r1, r2 = diameter[c["gid_i"]] / 2, diameter[c["gid_j"]] / 2
    fe = np.sqrt(r1 * r2 / (r1 + r2)) * KCC * over ** 1.5
    f = c["normal"] * fe[:, None]
    force, stress, size = np.zeros((n, 6)), np.zeros(n), np.zeros((n, 6))
    for g, s, r, w in (("gid_i", 1.0, "r_i", "stress_i"), ("gid_j", -1.0, "r_j", "stress_j")):
        terms = np.concatenate([s * f, np.cross(c[r], s * f)], axis=1)
        np.add.at(force, c[g], terms)
        np.add.at(size, c[g], np.abs(terms))
        np.add.at(stress, c[g], c[w] * fe)
    return force, stress, size


@pytest.mark.parametrize("n,m,hubs", [
    (1, 0, []), (1, 3, []), (2, 1, []), (31, 100, [7, 8, 9]), (32, 100, [31, 32, 33]), (33, 0, [200]),
    (2046, 6000, [64]), (2047, 6000, []), (2048, 6000, [40]), (2049, 6000, []), (20000, 64000, [33, 500]),
    (MAX_CELLS, MAX_CONTACTS - 300, [300])])
def test_noalloc_matches_plain_sum(n, m, hubs):
    import torch

    c = contacts(n, m, hubs, seed=n + m)
    diameter = np.random.default_rng(1).uniform(0.4, 0.6, n)
    dev = torch.device("cuda:0")
    t = {k: torch.as_tensor(np.ascontiguousarray(v), device=dev) for k, v in c.items()}
    d = torch.as_tensor(diameter, device=dev)
    force = torch.full((n, 6), float("nan"), dtype=torch.float64, device=dev)
    stress = torch.full((n,), float("nan"), dtype=torch.float64, device=dev)
    rc = _entry()(*[t[k].data_ptr() for k in ("gid_i", "gid_j", "sd", "normal", "r_i", "r_j", "stress_i", "stress_j")],
                  c["sd"].size, d.data_ptr(), n, KCC, force.data_ptr(), stress.data_ptr(),
                  torch.cuda.current_stream(dev).cuda_stream)
    assert rc == abi.PCC_OK
    want_f, want_s, size = plain(c, n, diameter)
    assert np.all(np.abs(force.cpu().numpy() - want_f) <= 1e-12 * size)
    np.testing.assert_allclose(stress.cpu().numpy(), want_s, rtol=1e-12, atol=0)
