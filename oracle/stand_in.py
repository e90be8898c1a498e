"""Closed-form stand-ins for the generated data files, for checkouts without them.

The colour tables derive from the CIE datasets and the OpenPBR tables from the upstream library's data;
neither is part of this repository, and both are generated where the reference is checked out
(`__graft_entry__.build`). Elsewhere the tests, the smoke check and the bench render with smooth stand-ins of the same
shapes: multi-lobe fits of the colour-matching functions (Wyman, Sloan and Shirley 2013), a 6504 K
Planckian illuminant, an energy table from the Schlick reflectance and a flat sheen fit. The GPU and the oracle get
the same tables, so what compares the two holds; what compares against the reference's data does not
(`tests/conftest.py` skips it).
"""
from __future__ import annotations

import functools
import math

import numpy as np

_XYZ_TO_RGB = np.array([[3.2404542, -1.5371385, -0.4985314], [-0.9692660, 1.8760108, 0.0415560], [0.0556434, -0.2040259, 1.0572252]])


def _cmf(lam):
    def lobe(mu, s1, s2):
        return np.exp(-0.5 * ((lam - mu) / np.where(lam < mu, s1, s2)) ** 2)
    x = 1.056 * lobe(599.8, 37.9, 31.0) + 0.362 * lobe(442.0, 16.0, 26.7) - 0.065 * lobe(501.1, 20.4, 26.2)
    y = 0.821 * lobe(568.8, 46.9, 40.5) + 0.286 * lobe(530.9, 16.3, 31.1)
    z = 1.217 * lobe(437.0, 11.8, 36.0) + 0.681 * lobe(459.0, 26.0, 13.8)
    return np.stack([x, y, z], 1)


def _planck(lam):
    return 1.0 / (lam ** 5 * np.expm1(1.4388e7 / (lam * 6504.0)))


@functools.lru_cache(maxsize=None)
def _spectral(lo: int, hi: int) -> dict:
    full, lam = np.arange(360, 831, dtype=np.float64), np.arange(lo, hi + 1, dtype=np.float64)
    weights = (_cmf(full) @ _XYZ_TO_RGB.T) * _planck(full)[:, None]
    weights = weights / weights.sum(0)                    # the illuminant maps to rgb (1, 1, 1)
    spd = _planck(lam) / (_cmf(lam)[:, 1] * _planck(lam)).sum()
    rgb = _cmf(lam) @ _XYZ_TO_RGB.T
    rgb = rgb / (rgb * spd[:, None]).sum(0)
    s = np.abs(rgb).sum(1)
    trapezoid = lambda v: (0.5 * (v[1:] + v[:-1])).sum()  # noqa: E731
    density = 0.9 * spd * s / trapezoid(spd * s) + 0.1 * s / trapezoid(s)
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * (density[1:] + density[:-1]))])
    icdf = np.interp(np.linspace(0, 1, 1025), cdf / cdf[-1], lam)
    visible = np.cumsum(_cmf(full).sum(1) + 0.01)         # a phase warp that spends itself where the eye sees
    phase = -math.pi + math.pi * (visible - visible[0]) / (visible[-1] - visible[0])
    return {"lambda_min": lo, "lambda_max": hi, "n": len(lam), "segments": 1024, "cmf_rgb": rgb.astype(np.float32),
            "illum": spd.astype(np.float32), "icdf": icdf.astype(np.float32), "xyz_to_rgb": _XYZ_TO_RGB,
            "uplift_w": np.ascontiguousarray(weights), "uplift_cos": np.cos(phase),
            "cos_phase": np.cos(np.interp(lam, full, phase)).astype(np.float32)}


def spectral_tables(lambda_min: int = 380, lambda_max: int = 780) -> dict:
    """As metal_vibe_tracer_b200.spectral_tables.load."""
    return {k: v.copy() if isinstance(v, np.ndarray) else v for k, v in _spectral(lambda_min, lambda_max).items()}


def openpbr_tables() -> dict:
    """As metal_vibe_tracer_b200.openpbr_tables.load."""
    n = 32
    at = (np.arange(n) + 0.5) / n
    f0 = (2.0 * at / (2.0 + 2.0 * at)) ** 2               # IOR 1 + 2 x
    albedo = f0[:, None, None] + (1 - f0[:, None, None]) * (1 - at[None, None, :]) ** 5 * (1 - 0.6 * at[None, :, None] ** 2)
    return {"opaque_energy": np.round(65535 * (1 - albedo)).astype(np.uint16).reshape(-1),
            "opaque_average": np.round(65535 * (1 - (2 * albedo * at).mean(2))).astype(np.uint16).reshape(-1),
            "ltc": np.tile(np.array([1.0, 0.0, 0.1], np.float32), n * n)}


def install() -> bool:
    """Has the package's load functions give the stand-ins where the generated files are missing;
    whether any is."""
    from metal_vibe_tracer_b200 import openpbr_tables as pbr, spectral_tables as spectral
    missing = False
    if not spectral.path().exists():
        spectral.load, missing = spectral_tables, True
    if not pbr.DATA.exists():
        pbr.load, missing = openpbr_tables, True
    return missing
