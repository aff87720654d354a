"""GPU tests of the sizes of the three-body blocks: the scratch of their numbering at counts beyond 32 bits."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_scan_scratch_grows_with_the_count():
    from dftd3 import library
    size = getattr(ctypes.CDLL(str(library._LIBPATH)), "_ZN2d319atm_scan_temp_bytesEx")    # d3::atm_scan_temp_bytes
    size.argtypes, size.restype = [ctypes.c_longlong], ctypes.c_size_t
    counts = [1 << 20, 10 ** 9, (1 << 31) - 2, (1 << 31) + 16, 5 * (1 << 29), 1 << 33]
    sizes = [size(n) for n in counts]
    assert 0 < sizes[0] < sizes[1] < sizes[2] <= sizes[3] < sizes[4] < sizes[5]


def _cells(nsys):
    """Crystals of nine atoms in seven lattices, one of 300 atoms among them; some 300 neighbours per atom."""
    import numpy as np
    from dftd3 import synthetic as S
    rng = np.random.default_rng(5)

    def cell(natoms, edge):
        lat = np.diag(rng.uniform(edge, 1.03 * edge, size=3))
        return rng.choice([1, 6, 8], size=natoms).astype(np.int32), S.pack_cell(rng, natoms, lat, 2.0), lat

    nine = [cell(9, 10.0) for _ in range(7)]
    big = cell(300, 26.0)
    return [big if k == nsys // 2 else nine[k % 7] for k in range(nsys)]


def _evaluate(systems, precision, graph=False, calls=1):
    import numpy as np
    from dftd3 import synthetic as S
    from dftd3.interface import BatchedDispersion, RationalDampingParam
    bat = BatchedDispersion([s[0] for s in systems], [s[1] for s in systems], np.array([s[2] for s in systems]),
                            np.ones((len(systems), 3), dtype=bool))
    bat.set_realspace_cutoff(9.0, 19.9, 9.0)
    bat.set_precision(precision)
    bat.set_graph(graph)
    param = RationalDampingParam(**{k: S.PBE_BJ[k] for k in ("s6", "s8", "a1", "a2", "alp")}, s9=1.0)
    for _ in range(calls):
        res = bat.get_dispersion(param, grad=True)
    return np.array(res["energy"]), res["gradient"], np.array(res["virial"])


@pytest.mark.parametrize("precision, graph, nsys", [("mixed", False, 345000), ("fp64", True, 60000)])
def test_batches_above_the_block_limit(precision, graph, nsys):
    """7.2e7 blocks within reach of the cutoff (more records than 32 bits number, 1e11 bytes) and 2.2e7 candidates,
    taken in groups of systems: every system as in a batch of eight (FP64 1e-12, the bound of the other three-body
    tests; FP32 2e-6, nine pair values of two units of 2^-24 each, twice)."""
    import numpy as np
    systems = _cells(nsys)
    e, g, v = _evaluate(systems, precision, graph, 2 if graph else 1)
    few = [systems[nsys // 2]] + [systems[k] for k in range(7)]
    e0, g0, v0 = _evaluate(few, precision)
    at = 1 + np.arange(nsys) % 7
    at[nsys // 2] = 0
    tol = 1.0e-12 if precision == "fp64" else 2.0e-6
    assert np.abs(e - e0[at]).max() <= tol * np.abs(e0[1:]).min()
    assert np.abs(v - v0[at]).max() <= tol * np.abs(v0).max()
    assert max(np.abs(x - g0[k]).max() for x, k in zip(g, at)) <= tol * np.abs(g0[0]).max()
