"""The step kernel's form on the CPU (the host engine against stand-ins for the
CUDA runtime): the block size and items that fn_get_stats reports, handed to
fn_set_kernel_shape or fn_create, give the form they were read from, on both
sides of the size up to which the default is five warps per 28 beads."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fibrenet_b200 import generate as g
from fibrenet_b200.model import PAIR_HS, Settings

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host_upload")
THREAD, STAGED, WIDE = range(3)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from fibrenet_b200 import build
    so = str(tmp_path_factory.mktemp("shape") / "libshape.so")
    out = subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-Xcompiler",
                          "-fPIC", "-include", os.path.join(HERE, "fake_cuda.h"), "-shared", "-o", so,
                          os.path.join(HERE, "shape_harness.cu")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-3000:]
    lib = C.CDLL(so)
    lib.hu_error.restype = C.c_char_p
    return lib


class Context:
    def __init__(self, lib, model, block_size=0):
        from fibrenet_b200 import native
        self.lib = lib
        self.h = C.c_void_p()
        assert lib.hs_create(block_size, C.byref(self.h)) == 0
        keep = native._Keep()
        desc = (native.FnNetworkDesc * 1)(native.network_desc(model, keep))
        assert lib.hu_upload(self.h, 1, desc) == 0, lib.hu_error(self.h)

    def form(self):
        return self.lib.hs_form(self.h)

    def shape(self):
        out = (C.c_int * 2)()
        self.lib.hs_shape(self.h, out)
        return tuple(out)

    def set_shape(self, block, items=0):
        assert self.lib.hs_set_shape(self.h, block, items) == 0, self.lib.hu_error(self.h)

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.lib.hu_destroy(self.h)


def fibres(beads, n):
    img = np.zeros((n, beads, 3))
    img[:, :, 0] = 1.0 + np.arange(beads)
    img[:, :, 1] = (1.0 + np.arange(n) % 250)[:, None]
    img[:, :, 2] = (1.0 + np.arange(n) // 250)[:, None]
    st = Settings(dt=0.001, cutoff=1.0, box_unit_cell=2.0, box=(beads + 2.0, 252.0, 12.0), bc_type=0)
    return g.chain_model(img, st, ["A"], [PAIR_HS], [[50.0, 0, 0, 0]])


@pytest.mark.parametrize("beads,n,form", [(10, 3, WIDE), (100, 500, WIDE), (97, 517, THREAD)])
def test_reported_shape_gives_the_form_again(lib, beads, n, form):
    assert (form == WIDE) == (beads * n <= 50_000)
    with Context(lib, fibres(beads, n)) as c:
        assert c.form() == form
        default = c.shape()
        for block, items, want in ((64, 0, THREAD), (96, 0, THREAD), (64, 2, STAGED), (256, 0, THREAD), (128, 4, STAGED)):
            c.set_shape(block, items)
            assert (c.shape(), c.form()) == ((block, items), want)
            c.set_shape(*default)
            assert (c.shape(), c.form()) == (default, form)
    with Context(lib, fibres(beads, n), block_size=default[0]) as c:
        assert (c.shape(), c.form()) == (default, form)
    with Context(lib, fibres(beads, n), block_size=192) as c:
        assert (c.shape(), c.form()) == ((192, 0), THREAD)
