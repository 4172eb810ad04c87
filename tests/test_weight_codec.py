"""The library's host codecs against the numpy form of the same arithmetic: every byte equal."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from raster_b200 import _lib as L
from raster_b200 import build
from raster_b200.quant import cpu_quant as cq

CODECS = {"q4_0": lambda w: cq.quantize_weight(w, cq.q4_0), "q8_0": lambda w: cq.quantize_weight(w, cq.q8_0),
          "q4_K": cq.quantize_weight_q4k, "q6_K": cq.quantize_weight_q6k}


def values(kind, n):
    rng = np.random.default_rng(3)
    w = rng.standard_normal(n).astype(np.float32)
    if kind == "zeros of both signs":
        w[: n // 2] = -0.0
    elif kind == "ties":
        w = np.round(w * 3) / 2
    elif kind == "subnormal":
        w *= np.float32(1e-42)
    elif kind == "wide range":
        w *= np.exp(rng.uniform(-80, 80, n))
    elif kind == "far from zero":
        w = 1000 + w * np.float32(1e-5)
    elif kind == "not finite":
        w[5], w[n // 2] = np.nan, np.inf
    return w.astype(np.float32)


@pytest.mark.parametrize("fmt", sorted(CODECS))
@pytest.mark.parametrize("kind", ["normal", "zeros of both signs", "ties", "subnormal", "wide range", "far from zero", "not finite"])
@pytest.mark.parametrize("n", [256, 256 * 515])   # one super-block; several threads with a remainder
def test_native_codec_gives_the_bytes_of_the_numpy_form(monkeypatch, fmt, kind, n):
    w = values(kind, n)
    with np.errstate(all="ignore"):
        got = CODECS[fmt](w)
        monkeypatch.setattr(cq, "_native", lambda *a, **k: None)
        want = CODECS[fmt](w)
    assert sorted(got) == sorted(want)
    for k in want:
        assert got[k].dtype == want[k].dtype and got[k].tobytes() == want[k].tobytes(), k
    with pytest.raises(ValueError):
        CODECS[fmt](w[:-1])


def test_codec_entry_points_check_their_arguments():
    lib = L.load()
    a = np.zeros(256, np.float32)
    p = a.ctypes.data
    assert lib.rstq_quantize_weight(None, p, p, 256, L.FMT_Q4_0) == L.E_INVALID
    assert lib.rstq_quantize_weight(p, p, p, 33, L.FMT_Q4_0) == L.E_SHAPE
    assert lib.rstq_quantize_weight(p, p, p, 32, L.FMT_Q8_S) == L.E_INVALID
    assert lib.rstq_quantize_weight_q4k(p, p, p, p, p, p, 128) == L.E_SHAPE
    assert lib.rstq_quantize_weight_q6k(p, p, p, None, 256) == L.E_INVALID


@pytest.fixture(scope="module")
def base_form(tmp_path_factory):
    """The codecs as a host without AVX2 (one that is no x86, for instance) compiles them."""
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    d = tmp_path_factory.mktemp("codec")
    (d / "c.cpp").write_text('#include "codec.cu"\nnamespace rstq { void set_error(const char*, ...) {} }\n')
    subprocess.run(["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-pthread", "-DRSTQ_NO_AVX2", "-I", build.CSRC, "-I", cuda,
                    "-I", os.path.join(build.HERE, "..", "include"), str(d / "c.cpp"), "-o", str(d / "c.so")], check=True)
    lib = C.CDLL(str(d / "c.so"))
    for n in ("rstq_quantize_weight", "rstq_quantize_weight_q4k", "rstq_quantize_weight_q6k"):
        getattr(lib, n).argtypes = L.SIGNATURES[n]
    return lib


@pytest.mark.parametrize("fmt", sorted(CODECS))
@pytest.mark.parametrize("kind", ["normal", "ties", "wide range", "far from zero"])
def test_base_form_gives_the_same_bytes(monkeypatch, base_form, fmt, kind):
    w = values(kind, 256 * 67)
    want = CODECS[fmt](w)
    monkeypatch.setattr(L, "load", lambda: base_form)
    got = CODECS[fmt](w)
    for k in want:
        assert got[k].tobytes() == want[k].tobytes(), k


@pytest.mark.parametrize("fmt", ["q4_0", "q8_0"])
def test_codec_next_to_its_ties(monkeypatch, fmt):
    """Codes are taken in f32 except near a tie: quotients within a few f32 steps of k + 0.5, on either side of it and
    of the line where the double path takes over, for scales over the normal range and beyond; and blocks whose
    largest magnitude occurs with both signs, in either order."""
    zp = 8 if fmt == "q4_0" else 128
    rng = np.random.default_rng(11)
    blocks = []
    for e in (-130, -101, -100, -30, 0, 40, 99, 100, 110):
        for _ in range(40):
            s = np.float32(rng.uniform(1, 2) * 2.0 ** (e - 7))
            k = rng.integers(-zp, zp, 32) + 0.5 + rng.choice([0, 1e-7, -1e-7, 1e-5, -1e-5, 9e-5, -9e-5, 1.1e-4, -1.1e-4], 32)
            b = (k * np.float64(s)).astype(np.float32)
            b[rng.permutation(32)[:2]] = np.float32(zp) * s * rng.choice([-1, 1], 2).astype(np.float32)
            blocks.append(b)
    w = np.concatenate(blocks)
    assert np.isfinite(w).all()
    got = CODECS[fmt](w)
    monkeypatch.setattr(cq, "_native", lambda *a, **k: None)
    want = CODECS[fmt](w)
    for k in want:
        assert got[k].tobytes() == want[k].tobytes(), k
