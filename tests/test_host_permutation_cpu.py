"""The host permutations against the oracle: random states, states of 0, 1 and
p - 1 in every mixture, one extreme word among zeros, and chains of outputs.
"""
import numpy as np
import pytest

import whir_gb300 as W

ONE = 0x01FFFFFE  # Montgomery form of 1


@pytest.mark.parametrize("width", [16, 24])
def test_extreme_states(oracle, width):
    rng = np.random.default_rng(width)
    states = [np.full(width, v, np.uint32) for v in (0, ONE, W.P - 1)]
    for lane in range(width):
        for v in (1, ONE, W.P - 1):
            s = np.zeros(width, np.uint32)
            s[lane] = v
            states.append(s)
    edge = np.array([0, 1, ONE, W.P - 1, (W.P - 1) // 2], np.uint32)
    states += [edge[rng.integers(0, 5, width)] for _ in range(400)]
    for s in states:
        assert np.array_equal(W.poseidon2_permute(width, s), oracle.p2_permute(width, s)), s


@pytest.mark.parametrize("width", [16, 24])
def test_chains(oracle, width):
    a = b = oracle.rand_fe(3, width)
    for _ in range(500):
        a, b = W.poseidon2_permute(width, a), oracle.p2_permute(width, b)
        assert np.array_equal(a, b)
