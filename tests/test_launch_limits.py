"""Launch shapes of the transforms against the shared-memory limits, without a GPU: the
library's own objects linked with a stand-in for the CUDA runtime (fake_cudart.cpp) that
refuses what the runtime would refuse.  The child process makes handles through the C ABI and
asks each for a potential; memory copies and kernels do nothing."""
import pytest

from fake_lib import fake_child, fake_lib  # noqa: F401 (a fixture)


CHILD = r"""
import ctypes as C, json
L = D.lib()
L.fake_max_smem.restype = C.c_size_t
bad, smem = [], 0
host = (C.c_double * 1)()
for Nu, Nphi, prec, dev in json.loads(arg):
    L.fake_reset()
    p = D.default_params(Nu=Nu, Nphi=Nphi, precision=prec, device=dev)
    h = C.c_void_p()
    rc = L.dg_create(C.byref(p), C.byref(h))
    if rc == 0:
        rc = L.dg_potential(h, host, host)
        L.dg_destroy(h)
    smem = max(smem, L.fake_max_smem())
    if rc or L.fake_refused():
        bad.append((Nu, Nphi, prec, dev, rc))
print(json.dumps([bad, smem]))
"""


def refused(lib, grids):
    return fake_child(lib, CHILD, grids)


def smooth(lo, hi):
    def ok(n):
        for p in (2, 3, 5):
            while n % p == 0:
                n //= p
        return n == 1
    return [n for n in range(lo, hi + 1) if ok(n)]


def test_every_accepted_length_launches(fake_lib):
    """Every length of either direction, beside few, some and many transforms of it."""
    grids = [(Nu, Nphi, "fp64", 0) for Nphi in smooth(2, 8192) for Nu in (6, 300, 4096)]
    grids += [(Nu, Nphi, "fp64", 0) for Nu in smooth(2, 4096) for Nphi in (9, 640, 8192)]
    grids += [(Nu, Nphi, "mixed", 0) for Nphi in smooth(2, 8192) if Nphi % 128 == 0
              for Nu in (128, 384, 640, 4096)]
    bad, smem = refused(fake_lib, grids)
    assert bad == []
    assert smem > 100 * 1024  # the stand-in saw the large transforms


def test_second_device_of_a_process(fake_lib):
    """The limits belong to a device: handles on the process's second and third one launch like
    those on the first (passes of more than 48 KB: u from 1350 points, phi in batches of rows,
    and the set-up transforms of a mixed disk)."""
    sizes = [(1350, 64, "fp64"), (4096, 9, "fp64"), (640, 1000, "fp64"), (6, 8192, "fp64"), (1024, 1024, "fp64"),
             (2048, 128, "mixed"), (256, 4096, "mixed"), (384, 8192, "mixed")]
    bad, smem = refused(fake_lib, [s + (dev,) for dev in (0, 1, 2) for s in sizes])
    assert bad == []
    assert smem > 48 * 1024


FAILS = r"""
import ctypes as C, json
L = D.lib()
host = (C.c_double * 1)()
out = []
for Nu, Nphi, prec in json.loads(arg):
    p = D.default_params(Nu=Nu, Nphi=Nphi, precision=prec)
    def go():
        h = C.c_void_p()
        rc = L.dg_create(C.byref(p), C.byref(h))
        if rc == 0:
            rc = L.dg_potential(h, host, host)
            L.dg_destroy(h)
        return rc
    L.fake_fail_at(C.c_longlong(-1))
    ok = go()
    n = L.fake_launches()
    for k in range(n):
        L.fake_fail_at(C.c_longlong(k))
        bad = go()
        L.fake_fail_at(C.c_longlong(-1))
        out.append((Nu, Nphi, prec, k, ok, bad, go()))
print(json.dumps(out))
"""


def test_a_failed_launch_is_reported_once(fake_lib):
    """A launch that the runtime refuses fails the call that made it and no later one."""
    rows = fake_child(fake_lib, FAILS, [(128, 128, "fp64"), (60, 90, "fp64"), (1152, 1152, "mixed")])
    assert len(rows) > 18
    for *what, ok, bad, after in rows:
        assert ok == 0 and bad == -2 and after == 0, (what, ok, bad, after)


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi,prec", [(300, 8192, "fp64"), (640, 6400, "fp64"), (405, 7500, "fp64"),
                                          (1000, 6250, "fp64"), (384, 8192, "mixed")])
def test_potential_of_many_long_rows(Nu, Nphi, prec):
    """The same on the GPU, values included: the bounds of the other potential tests over
    lengths, 1e-12 (FP64) and 1e-6 (FP32 transforms)."""
    import numpy as np

    import diskgpu as D
    import oracle as O
    from helpers import rel_err
    r = np.random.RandomState(Nu * 8209 + Nphi)
    Sig = r.uniform(0.1, 1.0, (Nu, Nphi))
    want = O.Kalnajs(Nu, Nphi, eps=0.01).potential(Sig)
    with D.Disk(Nu, Nphi, eps=0.01, precision=prec) as d:
        got = d.potential(Sig)
    assert rel_err(got, want) < (1e-12 if prec == "fp64" else 1e-6)
