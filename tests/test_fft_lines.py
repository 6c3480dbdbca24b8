"""The integer transforms of a line (tests/cpp/fft_lines.cpp) against numpy's
FP64 transform, both measured by numpy's extended-precision one, for each
size and each kind of line by itself: even and uneven, localised and
decaying ones.

Bound: the error (2-norm, root mean square over the lines of a kind) is at
most 1.1 times numpy's, the 0.1 for the spread over 24 lines, or 2^-53,
which rounding exact results to FP64 alone may cost."""
import os
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT

SIZES = (32, 40, 48, 64, 72, 80, 96, 100, 120, 128, 144, 160, 192, 200, 240, 256, 288, 320, 384)
LINES = 24


def kinds(P, rng):
    """name -> LINES lines of P complex values"""
    n = np.arange(P)

    def noise(scale=1.0):
        return scale * (rng.standard_normal((LINES, P)) + 1j * rng.standard_normal((LINES, P)))

    def at(width):
        c = rng.uniform(0, P, (LINES, 1))
        return np.exp(-0.5 * (((n - c + P / 2) % P - P / 2) / width) ** 2)

    one = noise(1e-3 / P)
    one[np.arange(LINES), rng.integers(0, P, LINES)] = noise()[:, 0]
    few = noise(1e-9)
    for q in range(LINES):
        few[q, rng.integers(0, P, 4)] = noise()[0, :4]
    phase = rng.uniform(0, 2 * np.pi, (LINES, 3, 1))
    half = noise()
    half[:, P // 2:] = 0
    out = {
        "noise": noise(),
        "even magnitudes": np.exp(2j * np.pi * rng.uniform(size=(LINES, P))),
        "even magnitudes near two": 1.99 * np.exp(2j * np.pi * rng.uniform(size=(LINES, P))),
        "smooth": sum(np.cos(2 * np.pi * (q + 1) * n / P + phase[:, q]) for q in range(3)) + 0j,
        "steep": noise() * np.exp(-20 * rng.uniform(size=(LINES, P))),
        "one large value": one,
        "few large values": few,
        "padded": half,
        "large and small": noise() * np.exp2(rng.integers(-300, 300, (LINES, 1))),
    }
    for d in (1.5, 6, 25, 100):
        out[f"decay over {d}"] = noise() * np.exp(-n / d)
        out[f"decay over {d}, real"] = noise().real * np.exp(-n / d) + 0j
    for w in (1, 3, 10):
        out[f"blob of width {w}"] = at(w) * np.exp(2j * np.pi * rng.uniform(size=(LINES, 1)))
        out[f"bubble wall of width {w}"] = 0.5 * (1 - np.tanh((np.abs(n - P / 2) - P / 8) / w)) * (
            1 + 1e-3 * noise())
    return out


def errors(lines, results):
    exact = np.fft.fft(lines.astype(np.clongdouble))
    d = np.abs(results - exact) ** 2
    return float(np.sqrt(np.mean(d.sum(1) / (np.abs(exact) ** 2).sum(1))))


@pytest.fixture(scope="module")
def transform(tmp_path_factory):
    if np.finfo(np.longdouble).nmant < 63 or \
            np.fft.fft(np.zeros(4, np.clongdouble)).dtype != np.clongdouble:
        pytest.skip("no extended-precision transform in numpy")
    exe = str(tmp_path_factory.mktemp("fft") / "fft_lines")
    inc = ["-I" + os.path.join(ROOT, *p) for p in (("sledgehamr_gb300", "csrc"), ("include",),
                                                   ("include", "sledgehamr"))]
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-w"] + inc +
                       [os.path.join(ROOT, "tests", "cpp", "fft_lines.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]

    def run(lines, *bits):
        z = np.ascontiguousarray(lines, dtype=np.complex128)
        r = subprocess.run([exe, str(z.shape[1]), str(z.shape[0]), *map(str, bits)],
                           input=z.tobytes(), capture_output=True)
        assert r.returncode == 0
        return np.frombuffer(r.stdout, dtype=np.complex128).reshape(z.shape)

    return run


@pytest.mark.parametrize("P", SIZES)
def test_every_kind_of_line_as_accurate_as_fp64(transform, P):
    bad = []
    for name, lines in kinds(P, np.random.default_rng(P)).items():
        here, fp64 = errors(lines, transform(lines)), errors(lines, np.fft.fft(lines))
        if not here <= max(1.1 * fp64, 2.0 ** -53):
            bad.append(f"{name}: {here:.2e}, numpy {fp64:.2e}")
    assert not bad, bad


def test_extreme_lines(transform):
    """Sums at the bounds: every value the largest there is below a power of
    two, in phase at some frequency; zeros; NaN-free scaling by powers of two
    is exact."""
    for P in SIZES:
        n = np.arange(P)
        top = np.nextafter(2.0, 0)
        rows = [top * (1 + 1j) * np.ones(P), np.zeros(P, complex), top * (1 - 1j) * (-1.0) ** n]
        rows += [top * np.exp(2j * np.pi * k * n / P) for k in range(0, P, max(1, P // 16))]
        rows += [np.sign(np.cos(2 * np.pi * k * n / P) + 1e-3) * top * (1 + 1j)
                 for k in range(1, P // 2, max(1, P // 16))]
        lines = np.array(rows)
        got = transform(lines)
        scale = P * np.abs(lines).max()
        assert np.all(np.abs(got - np.fft.fft(lines)) <= 4e-15 * scale)
        assert np.array_equal(transform(lines * 2.0 ** -200), got * 2.0 ** -200)
