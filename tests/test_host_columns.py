"""CPU checks of the on-chip sweep's band plans (no GPU): what the kernel
relies on, over grids of all shapes, cluster sizes and threads per column."""
import pytest

import x2dhf_gb300 as xg

SMEM_MOST = 227 * 1024
GRIDS = [(31, 31), (61, 31), (31, 61), (91, 121), (121, 331), (151, 241), (331, 481), (361, 571), (511, 301), (151, 811),
         (271, 811), (241, 901), (181, 1201), (91, 1831), (541, 31), (781, 31)]


def _plans(nnu, nmu):
    for size in range(1, 17):
        for groups in (1, 2):
            p = xg.host_column_plan(nnu, nmu, size, groups)
            if p:
                yield size, groups, p


@pytest.mark.parametrize("nnu,nmu", GRIDS)
def test_bands_cover_the_rows_and_hold_their_points(nnu, nmu):
    """Bands cover the interior rows 5..nmu-1 one after the other, at least 8
    rows each (halos of four rows come from the next band alone, and a halo's
    rows from one thread); the row seam lies inside one thread's rows, five or
    more below and ten above it; no thread has more points of a colour (every
    fifth row, counted on each side of the seam) than the plan's slots."""
    seam = (nmu + 7) // 2
    found = 0
    for size, groups, p in _plans(nnu, nmu):
        found += 1
        r = p["row0"]
        assert r[0] == 5 and r[-1] == nmu
        heights = [b - a for a, b in zip(r, r[1:])]
        assert min(heights) >= 8 and max(heights) == p["maxrows"]
        for k, n in enumerate(heights):
            cuts = [0, p["cut"][k], n] if groups == 2 else [0, n]
            assert cuts[1] >= 4 and n - cuts[-2] >= 4
            for a, b in zip(cuts, cuts[1:]):
                a, b = r[k] + a, r[k] + b
                assert seam not in (a, b)
                parts = [seam - a, b - seam] if a < seam < b else [b - a]
                if len(parts) == 2:
                    assert parts[0] >= 5 and parts[1] >= 10
                assert sum((x + 4) // 5 for x in parts) <= p["slots"]
    assert found > 0


@pytest.mark.parametrize("nnu,nmu", GRIDS)
@pytest.mark.parametrize("potentials", [0, 1, 2])
def test_kernels_hold_their_plans(nnu, nmu, potentials):
    """A kernel has at least the plan's slots, rows for every thread to go
    through all of its own slots, and fits an SM."""
    for size, groups, p in _plans(nnu, nmu):
        q = xg.host_column_plan(nnu, nmu, size, groups, potentials)
        if q["kernel_slots"] == 0:
            assert q["smem"] == 0
            continue
        assert q["kernel_slots"] >= q["slots"]
        last = max(q["cut"]) if groups == 2 else 0
        assert q["kernel_rows"] >= max(q["maxrows"], last + 5 * q["kernel_slots"]) + 4


# every grid size that one cluster held with bands of whole tiles: x2g_host_cluster_plan still says which those are
@pytest.mark.parametrize("nnu", [31, 61, 91, 121, 151, 181, 211, 241, 271, 301, 331])
def test_grids_that_one_cluster_held_are_still_on_chip(nnu):
    """Few columns and up to sixteen CTAs' rows (1:20), plain and potentials."""
    for nmu in range(31, min(2431, 20 * nnu) + 1, 30 if nnu > 250 else 240):
        if xg.host_cluster_plan(nnu, nmu)[0] == 0:
            continue
        for potentials in (0, 1):
            fits = [q for size, groups, p in _plans(nnu, nmu)
                    for q in [xg.host_column_plan(nnu, nmu, size, groups, potentials)]
                    if q["kernel_slots"] and q["smem"] <= SMEM_MOST]
            assert fits, (nnu, nmu, potentials)


@pytest.mark.parametrize("nnu", [511, 541, 661, 781])
def test_flat_grids_are_still_on_chip(nnu):
    assert xg.host_cluster_plan(nnu, 31)[0] > 0
    for potentials in (0, 1):
        assert any(q["kernel_slots"] and q["smem"] <= SMEM_MOST for size, groups, p in _plans(nnu, 31)
                   for q in [xg.host_column_plan(nnu, 31, size, groups, potentials)])
