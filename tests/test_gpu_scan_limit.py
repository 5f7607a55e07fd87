"""A prefix scan of the collider that gives up a wait (k_scan): the call that runs into it returns WDEM_ERR_TIMEOUT,
no kernel indexes by the half-scanned values, the handle stays readable with an empty container, and the device is
intact.  The waits are made to run out by allowing them no look at all, in a build of the engine with an accessor for
that limit; only scans of more than one tile (4096 values) wait."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from woo_gb300 import abi, build, scenes

from helpers import gpu_handle, gpu_particles

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def limited(wdem_lib, tmp_path_factory):
    names = [os.path.splitext(s)[0] for s in build.SOURCES if s != "wdem_api.cu"] + [v[1] for v in build.VARIANTS]
    objs = [os.path.join(build.BUILD, n + ".o") for n in names]
    if not all(map(os.path.exists, objs)):
        build.build(force=True)
    out = str(tmp_path_factory.mktemp("scan") / "libscanlimit.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-I", build.INCLUDE, "-shared",
                    os.path.join(HERE, "native", "scan_limit.cu"), *objs, "-o", out, "-lcudart"], check=True)
    return abi.load(out)


def _broken(h, call):
    with pytest.raises(abi.WdemError, match="prefix sum") as ei:
        call()
    assert ei.value.code == abi.WDEM_ERR_TIMEOUT


def _limit(lib, h, looks):
    lib.scan_limit_set.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.scan_limit_set(h.h, looks)


def _spec(kind):
    if kind == "peri":
        return scenes.periodic_cloud(5000, 1, size=(0.22, 0.22, 0.22))
    if kind == "carry":  # buckets and rows fit one tile, the pairs do not
        return scenes.random_cloud(1900, 1, box=(0.15, 0.15, 0.15), dense=0.8, verletDist=0.002)
    return scenes.random_cloud(5000, 1, box=(0.22, 0.22, 0.22), dense=0.85, trackEnergy=int(kind == "energy"))


@pytest.mark.parametrize("kind", ["buckets", "peri", "carry", "energy"])
@pytest.mark.parametrize("steps", [1, 40])
def test_step_reports_a_scan_that_gave_up(limited, monkeypatch, kind, steps):
    monkeypatch.setattr(abi, "_lib", limited)
    spec = _spec(kind)
    n = spec.particles.n
    assert n > (4096 if kind != "carry" else 0) and (kind != "carry" or n < 2040)
    h = gpu_handle(spec)
    _limit(limited, h, 0)
    _broken(h, lambda: h.step(steps))
    _broken(h, lambda: h.step(1))
    assert h.status().nContacts == 0 and h.download_contacts().n == 0
    p = gpu_particles(h, n)
    assert np.isfinite(p.pos).all() and np.isfinite(p.force).all()
    if kind == "peri":
        assert (np.asarray(h.stress()) == 0).all()
    h.remove_particles([n - 1])
    h.close()
    # a handle of its own on the same device runs the same scene
    h = gpu_handle(spec)
    h.step(steps)
    assert h.status().nContacts > (4096 if kind == "carry" else 0)
    h.close()


def test_uploaded_contacts_and_boxes(limited, monkeypatch):
    monkeypatch.setattr(abi, "_lib", limited)
    spec = _spec("buckets")
    h = gpu_handle(spec)
    h.step(5)
    c = h.download_contacts()
    assert c.n > 4096
    _limit(limited, h, 0)
    _broken(h, lambda: h.upload_contacts(c))
    assert h.download_contacts().n == 0
    h.close()
    h = abi.Handle(5000)
    _limit(limited, h, 0)
    lo = np.random.default_rng(0).uniform(0, 1, (5000, 3))
    _broken(h, lambda: h.collide_boxes(lo, lo + 0.05, np.full(5000, 5, np.uint32), 2))
    h.close()
