"""The table and the coefficients in csrc/gauss64.cuh are those of their definitions."""
import os
import re

from oracle import gauss_tables as G

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "thermal_inflation_phase_transition_b200", "csrc", "gauss64.cuh")


def source():
    with open(SRC) as f:
        return f.read()


def test_log_table():
    rows = [(int(a, 16), int(b, 16)) for a, b in re.findall(r"\{0x([0-9a-f]{16}), 0x([0-9a-f]{16})\}", source())]
    assert rows == G.log_table()


def test_log_step():
    head, rest = G.log_step()
    s = source()
    assert float.fromhex(re.search(r"head = __fma_rn\(k, (\S+),", s)[1]) == head
    assert float.fromhex(re.search(r"tail = __fma_rn\(k, (\S+),", s)[1]) == rest


def test_sine():
    body = source().split("double sin_half_pi(double y) {")[1].split("}")[0]
    got = [float.fromhex(x) for x in re.findall(r"-?0x1\.[0-9a-f]+p[+-]\d+", body)]
    assert got == G.sine()
