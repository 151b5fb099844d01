"""PGSR per-Gaussian plane descriptor ``all_map`` = [normal in camera space (3), 1, plane distance] as a
differentiable op: what the reference's caller builds with a dozen tensor operations right before
``render_gaussians`` (gaussian_renderer/__init__.py:1501-1518) is one kernel forward and one kernel backward here.

Gradients flow to ``means3D`` (through the distance) and to the raw quaternions (through the chosen rotation
column and ``normalize``); ``scales`` only select the column and receive none, exactly as in the reference's graph.
Rows with ``radii <= 0`` (never rasterized) are zero in both directions.
"""
from __future__ import annotations

from diff_gaussian_rasterization import _lib


def plane_map(means3D, scales, rotations, viewmatrix, campos, radii=None):
    """(P,5) all_map for one camera.  viewmatrix: the (4,4) row-vector world-to-view matrix of the rasterizer
    settings; campos: (3,).  radii (optional int32 (P)): rows with radius <= 0 are skipped."""
    return _lib.host().plane_map(means3D, scales, rotations, radii, viewmatrix, campos)
