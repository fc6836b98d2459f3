"""Trajectories in batches on the device: the same values whether a
trajectory runs alone or beside others, at the edges of a batch (64
trajectories), of the chunked norm (one chunk up to 12 qubits) and of the
tiles (gate by gate below 4 qubits), against the reference's loop restated
over the oracle's kernels (branches by cumulative Re Tr(K^dagger K rho),
the sequential norm)."""
import math

import numpy as np
import pytest

import pyoracle
from menos_b200 import Circuit
from menos_b200._lib import MB2Error
from menos_b200.engine import trajectories
from test_dm import noisy_circuit
from test_trajectories import trajectory_seed

pytestmark = pytest.mark.gpu


def restated(oracle, circ, count, seed, paulis, targets):
    """Term values per trajectory and the outcome of each one's shot."""
    n = circ.num_qubits
    values, shots = [], []
    for t in range(count):
        draws = iter(oracle.uniforms(trajectory_seed(seed, t), 256))
        psi = np.zeros(1 << n, np.complex128)
        psi[0] = 1.0
        for oc, qs, ps, m, _cl in circ.ops:
            if oc == pyoracle.OP["measure"]:
                continue
            if oc != pyoracle.OP["channel"]:
                oracle.apply_generic(psi, m if m is not None else oracle.gate_matrix(oc, ps), list(qs))
                continue
            k, dim = len(qs), 1 << len(qs)
            off = [sum(1 << qs[j] for j in range(k) if (a >> j) & 1) for a in range(dim)]
            base = np.array([b for b in range(1 << n) if not b & off[-1]])
            v = np.stack([psi[base | o] for o in off])
            rho = v @ v.conj().T
            u, cum, branch, last = next(draws), 0.0, None, None
            for i, kmat in enumerate(m):
                p = np.trace(kmat.conj().T @ kmat @ rho).real
                if p > 0.0:
                    last, cum = i, cum + p
                    if u < cum:
                        branch = i
                        break
            oracle.apply_generic(psi, m[last if branch is None else branch], list(qs))
            p = psi.real * psi.real + psi.imag * psi.imag
            psi = psi * (1.0 / math.sqrt(np.add.accumulate(p)[-1]))
        values.append([oracle.expectation(psi, x, z) for x, z in paulis])
        p = psi.real * psi.real + psi.imag * psi.imag
        b = min(int(np.searchsorted(np.add.accumulate(p), next(draws), side="right")), (1 << n) - 1)
        shots.append(sum(((b >> q) & 1) << c for q, c in targets))
    return np.array(values), shots


@pytest.mark.parametrize("n,count,widest", [(1, 5, 1), (3, 9, 3), (4, 70, 2), (7, 129, 3), (12, 6, 2), (13, 5, 3)])
def test_batches_are_the_trajectories_one_by_one(ctx, oracle, n, count, widest):
    rng = np.random.default_rng(n)
    c, d = noisy_circuit(n, 24, rng, widest=widest)
    paulis = [(int(x), int(z)) for x, z in rng.integers(0, 1 << n, size=(5, 2))] + [(0, 0)]
    targets = [(q, n - 1 - q) for q in range(n)]
    got = trajectories(ctx, d, count, 31, paulis, None, count, targets)
    want, shots = restated(oracle, c, count, 31, paulis, targets)
    assert np.max(np.abs(got["terms"] - want.mean(0))) < 1e-12
    total = want.sum(1)
    error = math.sqrt(sum(abs(v - total.mean()) ** 2 for v in total) / (count - 1) / count)
    assert abs(got["standard_error"] - error) <= 1e-9 * max(1.0, error)
    assert got["counts"].to_dict() == {o: shots.count(o) for o in sorted(set(shots))}
    # Fewer trajectories: the first ones' values, whatever ran beside them.
    few = trajectories(ctx, d, 2, 31, paulis)
    assert np.max(np.abs(few["terms"] - want[:2].mean(0))) < 1e-12


def test_refusals(ctx):
    dead = Circuit(5)
    dead.gate("h", [0])
    dead.channel([1], np.zeros((2, 2, 2)))  # no branch has a probability
    with pytest.raises(MB2Error, match="probability 0"):
        trajectories(ctx, dead, 70, 1, [(0, 1)])
    twice = Circuit(5)
    twice.channel([2, 2], np.eye(4)[None])
    with pytest.raises(MB2Error):
        trajectories(ctx, twice, 2, 1, [(0, 1)])
    fine = Circuit(5)
    fine.gate("h", [0])
    with pytest.raises(MB2Error):
        trajectories(ctx, fine, 2, 1, [(1 << 5, 0)])
    assert abs(trajectories(ctx, fine, 2, 1, [(1, 0)])["terms"][0] - 1.0) < 1e-12
