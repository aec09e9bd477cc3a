"""Which sectors of a blockwise SVD go to the cluster launch (``linalg.cluster_sectors``)."""

import pytest

from tenet import linalg

SMEM = (227 * 1024 - 1024) // 8


def _count(r, c):
    """Clusters at once, roughly as on a B200: an SM holds two to eight CTAs."""
    if r > 512 or c > 256:
        return 0
    pairs = max(1, (c + 1) // 2)
    cl = 1
    while cl < 16 and pairs > 4 * cl:
        cl *= 2
    return 148 * (8 if r <= 64 else 4 if r <= 128 else 2) // cl


@pytest.mark.parametrize("shapes, clustered", [
    ([(116, 116), (40, 30), (5, 1)], "all"),
    ([(64, 2), (40, 40)], "all"),        # a thin sector costs nothing beside another
    ([(512, 10)], []), ([(64, 2), (300, 20), (128, 4)], []),
    ([(512, 10), (64, 64)], [(64, 64)]),  # shorter columns for the others
    ([(512, 10), (400, 64)], "all"),      # none to be had
    ([(192, 20)] * 148, []), ([(96, 32)] * 300, []), ([(24, 24)] * 250, "all"),
    ([(48, 48)] * 150, "all"),
    ([(256, 256), (300, 300)], []), ([(512, 10), (300, 300)], [(512, 10)]),
    ([(64, 64), (256, 256), (300, 300)], [(64, 64)]),
    ([(256, 256), (300, 300)] * 80, [(256, 256)] * 80),
    ([(600, 4), (128, 128)], [(128, 128)]), ([(600, 20), (64, 64)], [(64, 64)]),
    ([(300, 257)], []), ([(512, 256)], "all"), ([(1, 1)], "all"), ([], "all")])
def test_cluster_sectors(shapes, clustered):
    got = linalg.cluster_sectors(dict(enumerate(shapes)), _count, SMEM)
    assert sorted(got.values()) == sorted(shapes if clustered == "all" else clustered)
    assert all(shapes[k] == x for k, x in got.items())
