"""Neighbour rows where the order of the search template can go wrong: cells
of very different sides (many offsets of equal or almost equal distance after
scaling), neighbourhoods wider than the grid (mirrored offsets of one row and
the next), rotated ellipsoids, one-cell axes and a template of one pair."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu

CASES = {
    "nearest_2d": ((23, 17), (1.0, 1.0), None, 12),
    "nearest_narrow": ((3, 90), (1.0, 1.0), None, 9),
    "flat_cells": ((40, 30), (1e-3, 1e3), None, 10),
    "tiny_against_huge": ((30, 6), (1e-9, 1e9), None, 14),
    "ball_over_the_grid": ((9, 11, 7), (1.0, 0.5, 2.0), geosgs.MetricBall(60.0), 20),
    "ellipsoid": ((15, 13, 9), (1.0, 1.0, 1.0), geosgs.MetricBall((7.0, 5.0, 3.0), geosgs.RotZ(30.0)), 16),
    "ellipsoid_uneven": ((25, 21), (0.37, 1.91), geosgs.MetricBall((6.0, 11.0)), 11),
    "one_row": ((64, 1), (1.0, 1.0), geosgs.MetricBall(9.0), 6),
    "one_pair": ((12, 9), (1.0, 3.0), geosgs.MetricBall(1.0), 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_neighbours_in_template_order(geosgs_lib, oracle_mod, name):
    dims, spacing, ball, k = CASES[name]
    grid = geosgs.CartesianGrid(dims, spacing=spacing)
    process = geosgs.GaussianProcess(geosgs.ExponentialVariogram(range=5.0, sill=1.0, nugget=0.1), 0.0)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(2), maxneighbors=k, precision="fp64", neighborhood=ball)
    p, keep = geosgs.build_problem(process, grid, None, method)
    plan = geosgs.Plan(p, keep).prepare()
    got, gcount = plan.neighbors()
    want, wcount = oracle_mod.OraclePlan(p, keep).prepare().neighbors()
    plan.close()
    np.testing.assert_array_equal(gcount, wcount)
    np.testing.assert_array_equal(got, want)
