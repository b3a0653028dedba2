"""Device-resident fields: boundary round trip and the Field reductions
(Field::norm, include/field.h:74-78; Field::operator*, lib/Fields/field.inl:58-62)."""
import threading

import numpy as np
import pytest

import iroiro_b200 as ib
from conftest import TOL_FP16, TOL_FP32, TOL_FP64

pytestmark = pytest.mark.gpu

L = [8, 8, 8, 16]
V = int(np.prod(L))


@pytest.fixture(scope="module")
def ctx():
    return ib.context(L)


@pytest.mark.parametrize("subset", [0, 1, 2])
def test_round_trip_is_bit_exact_in_fp64(ctx, subset):
    n = (24 if subset == 2 else 12) * V
    f = ib.synth_gaussian(n // 24, 81 + subset)
    d = ib.DeviceField(ctx, subset, "double").upload(f)
    assert np.array_equal(d.download(), f)


@pytest.mark.parametrize("prec,tol", [("double", TOL_FP64), ("single", TOL_FP32), ("half", TOL_FP16)])
def test_norm_and_dot(ctx, prec, tol):
    nrhs = 3
    a = ib.synth_gaussian(V * nrhs, 91)
    b = ib.synth_gaussian(V * nrhs, 92)
    da = ib.DeviceField(ctx, 2, prec, nrhs).upload(a)
    db = ib.DeviceField(ctx, 2, prec, nrhs).upload(b)
    A, B = a.reshape(nrhs, -1), b.reshape(nrhs, -1)
    assert np.allclose(da.norm(), np.linalg.norm(A, axis=1), rtol=tol, atol=0)
    ref = np.einsum("ri,ri->r", A, B)
    assert np.all(np.abs(da.dot(db) - ref) <= tol * np.linalg.norm(A, axis=1) * np.linalg.norm(B, axis=1))


@pytest.mark.parametrize("nrhs", [2, 3, 5, 12, 13])
def test_pageable_round_trip_around_the_threaded_copy(nrhs):
    """Uploads and downloads below and above the sizes from which pageable
    memory is copied by several threads in 1 MiB pieces (3 MiB per right-hand
    side here: direct copies, then pieces in one direction or both),
    bit for bit; again with two contexts copying from two threads at once."""
    L = [8, 8, 8, 32]
    n = int(np.prod(L)) * nrhs
    f = ib.synth_gaussian(n, 50 + nrhs)
    ctxs = [ib.Context(L, 0) for _ in range(2)]
    fields = [ib.DeviceField(c, 2, "double", nrhs) for c in ctxs]
    assert np.array_equal(fields[0].upload(f).download(), f)
    bad = []

    def work(k):
        g = f + k
        for _ in range(4):
            if not np.array_equal(fields[k].upload(g).download(), g):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_upload_with_work_queued_before_another_context_copies():
    """An upload whose DMAs wait behind work queued on its context, then copies
    of a second context of the device: the first context's field is what was
    uploaded, bit for bit."""
    L = [8, 8, 8, 32]
    V = int(np.prod(L))
    u = ib.synth_gauge(L, 0.2, 61, gauge_transform=True)
    a, b = ib.Context(L, 0), ib.Context(L, 0)
    a.upload_gauge(u)
    op = ib.Dirac_Wilson(0.5 / 0.12 - 4.0, u, ctx=a)
    f, g = ib.synth_gaussian(V * 11, 62), ib.synth_gaussian(V * 12, 63)
    fa, fb = ib.DeviceField(a, 2, "double", 11), ib.DeviceField(b, 2, "double", 12).upload(g)
    src, dst = (ib.DeviceField(a, 2, "double", 12).upload(g) for _ in range(2))
    for _ in range(20):
        for _ in range(50):  # a few ms
            a.check(ib.lib().iro_dirac_apply_field(a.h, op.op, op.mass, 0.0, 0, src.h, dst.h), "apply")
        fa.upload(f)
        assert np.array_equal(fb.download(), g)
        assert np.array_equal(fa.download(), f)
