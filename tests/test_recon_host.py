"""The PDM reconstruction of a face (gop_device.cuh), compiled for the host,
against PDMU7 as the reference writes it (src/solver_func.c:215-253), restated
here with numpy in 64 bits: random lines, ties, and the faces where something is
not finite.

Tolerance: a state is a sum of seven products and about six more operations, each
rounding 1.1e-16 (6e-8) of values of a few units: 1e-14 (6e-6) of the largest
magnitude in the line."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def _compile(tmp, axis):
    so = tmp / f"librecon{axis}.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-fPIC", "-shared", f"-DRECON_AXIS={axis}",
                    "-I/usr/local/cuda/include", f"-I{ROOT / 'gamera-op_b200/csrc'}",
                    str(ROOT / "tests/fake/recon_host.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("recon")
    return [_compile(tmp, axis) for axis in range(3)]


def _device(lib, bits, v, lim, w):
    out = np.zeros((len(v), 2))
    p = [np.ascontiguousarray(a, np.float64) for a in (v, lim, w)]
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    getattr(lib, f"recon{bits}")(len(v), *[ptr(a) for a in p], ptr(out))
    return out


def _sgn(x):
    return np.where(x > 0, 1.0, np.where(x < 0, -1.0, 0.0))


def _pdmu7(fi, near, far, opp, c1, c2):
    """One state: the value fi at the face, the cell it belongs to (near), that
    cell's other neighbour (far), the cell across (opp).  fmin and fmax pass over
    what is not a number."""
    lo, hi = np.fmin(near, opp), np.fmax(near, opp)
    f = np.fmax(lo, np.fmin(fi, hi))
    d0, d1 = near - far, opp - near
    q = np.abs(_sgn(d0) + _sgn(d1)) * (0.5 * np.abs(c1 * near + c2 * far) * 0.5 + 0.5 * np.abs(d0))
    return f - _sgn(d1) * np.fmax(0.0, np.abs(f - near) - q)


def _reference(v, lim, w):
    with np.errstate(invalid="ignore", over="ignore"):
        fl, fr = v[:, 0] * w[:, 0], v[:, 7] * w[:, 7]
        for t in range(1, 7):
            fl = fl + v[:, t] * w[:, t]
            fr = fr + v[:, 7 - t] * w[:, 7 + t]
        L = _pdmu7(fl, lim[:, 1], lim[:, 0], lim[:, 2], w[:, 14], w[:, 15])
        R = _pdmu7(fr, lim[:, 2], lim[:, 3], lim[:, 1], w[:, 16], w[:, 17])
    return np.stack([L, R], 1)


FAC = np.array([-1 / 140, 5 / 84, -101 / 420, 319 / 420, 107 / 210, -19 / 210, 1 / 105])


def _lines(rng, n, whole):
    """Half-step lines, their step-start limiters, weights (a stretched grid's)."""
    lim8 = rng.integers(-2, 3, (n, 8)).astype(float) if whole else rng.standard_normal((n, 8))
    v = lim8 + (0.0 if whole else 0.2) * rng.standard_normal((n, 8))
    w = np.concatenate([np.tile(FAC, (n, 2)), np.tile([2.0, -2.0, 2.0, -2.0], (n, 1))], 1)
    if not whole:
        w *= 1.0 + 0.1 * rng.standard_normal(w.shape)
    return v, lim8[:, 2:6], w


def _check(lib, v, lim, w):
    ref = _reference(v, lim, w)
    size = np.maximum(np.nan_to_num(np.abs(v), posinf=0.0).max(1), np.abs(lim).max(1))[:, None]
    for bits, tol in ((64, 1e-14), (32, 6e-6)):
        got = _device(lib, bits, v, lim, w)
        ok = np.abs(got - ref) <= tol * size
        if bits == 32:  # (a tie or a sign change may fall the other way in 32 bits)
            assert ok.mean() > 0.999
        else:
            assert ok.all(), (v[~ok.all(1)][0], lim[~ok.all(1)][0], got[~ok.all(1)][0], ref[~ok.all(1)][0])


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("whole", [False, True])
def test_states_of_a_face(libs, axis, whole):
    _check(libs[axis], *_lines(np.random.default_rng(axis), 20000, whole))


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("signs", [(1, 1), (1, -1), (-1, 1)])
def test_face_without_an_area(libs, signs, whole):
    """The theta face on a pole has no area: the limiter's coefficients, quotients
    by it, are infinite and what they multiply infinite or no number.  Then
    nothing is taken off the clamped value, whatever the signs of the slopes."""
    v, lim, w = _lines(np.random.default_rng(7), 20000, whole)
    w[:, 14], w[:, 15] = signs[0] * np.inf, signs[1] * np.inf
    w[:, 16], w[:, 17] = signs[1] * np.inf, signs[0] * np.inf
    _check(libs[1], v, lim, w)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("taps", [(0,), (7,), (3, 4), range(8)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("whole", [False, True])
def test_lost_taps(libs, axis, taps, value, whole):
    """A half-step value that is no number: the clamp's fmin leaves the larger of
    the two neighbours, on either side of the face and for either direction.  An
    infinite one is clamped."""
    v, lim, w = _lines(np.random.default_rng(11), 20000, whole)
    v[:, list(taps)] = value
    _check(libs[axis], v, lim, w)
