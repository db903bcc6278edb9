"""CPU checks of the drop-in boundary: the shared library loads without a GPU, exports
every symbol that include/b200mat.h declares (and nothing undeclared), the Python
structs match the C layout, and an operation without a device fails loudly."""
import ctypes as ct
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "b200mat.h")
LIB = os.path.join(ROOT, "deepnet_b200", "libb200mat.so")


def declared_functions():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = re.findall(r"^\s*(?:const\s+)?(?:unsigned\s+)?(?:int|void|float|char)\s*\*?\s*(\w+)\s*\(", text, flags=re.M)
    return sorted(set(names))


def test_header_compiles_as_c():
    subprocess.check_call(["gcc", "-std=c99", "-fsyntax-only", "-x", "c", HEADER])


def test_library_exports_every_declared_symbol():
    assert os.path.exists(LIB), "build the library first (python -m deepnet_b200.build)"
    lib = ct.CDLL(LIB)
    names = declared_functions()
    assert len(names) > 100
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, missing


def test_no_undeclared_exports():
    out = subprocess.check_output(["nm", "-D", "--defined-only", LIB], text=True)
    exported = {l.split()[-1] for l in out.splitlines() if " T " in l and not l.split()[-1].startswith("_")}
    extra = sorted(exported - set(declared_functions()))
    assert not extra, extra


def test_struct_layouts_match_header():
    from deepnet_b200 import b200mat
    assert ct.sizeof(b200mat.cudamat) == 40          # cudamat/cudamat.cuh:21-29 on LP64
    assert ct.sizeof(b200mat.rnd_struct) == 16       # same size as the reference's two pointers
    assert b200mat.cudamat.size.offset == 24 and b200mat.cudamat.is_trans.offset == 32
    code = r'''
#include <stdio.h>
#include "b200mat.h"
int main(void) { printf("%zu %zu %zu %zu\n", sizeof(cudamat), sizeof(rnd_struct), sizeof(b200_pass), sizeof(b200_fused_gemm)); return 0; }
'''
    exe = "/tmp/b200mat_abi_probe"
    subprocess.run(["gcc", "-x", "c", "-", "-I", os.path.join(ROOT, "include"), "-o", exe], input=code, text=True, check=True)
    sizes = [int(x) for x in subprocess.check_output([exe], text=True).split()]
    assert sizes == [ct.sizeof(b200mat.cudamat), ct.sizeof(b200mat.rnd_struct), ct.sizeof(b200mat._Pass),
                     ct.sizeof(b200mat._FusedGemm)]


def test_no_device_is_a_loud_failure_not_a_fallback():
    from deepnet_b200 import b200mat
    lib = ct.CDLL(LIB)
    if lib.b200_device_count() > 0:
        pytest.skip("a device is present")
    with pytest.raises(b200mat.CUDAMatException):
        b200mat.empty((2, 2))


def test_product_does_not_import_the_oracle():
    pkg = os.path.join(ROOT, "deepnet_b200")
    for dirpath, _, files in os.walk(pkg):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h")):
                text = open(os.path.join(dirpath, f)).read()
                assert "eigenmat_oracle" not in text and "liboracle" not in text, f


@pytest.mark.parametrize("shapes", [[(46341, 46341), (4, 4), (100000, 21475), (5, 1)], [(1 << 15, 1 << 15), (1, 64)], [(3, 5), (7, 7)]])
def test_matrices_beyond_a_column_get_an_allocation_of_their_own_shape(shapes, monkeypatch):
    """Matrices of 2^30 elements and more that share device memory: no allocation has a dimension beyond 2^31, every matrix lies
    inside one and over no other (on a stand-in that records what would be allocated)."""
    from deepnet_b200 import b200mat as cm

    class Stand(object):
        def __init__(self, shape, slab=None, first=0):
            assert 0 < shape[0] < 1 << 31 and 0 < shape[1] < 1 << 31
            self.shape, self.slab, self.first = shape, slab or self, first

        def slice(self, first, last):
            assert self.shape[1] == 1 and last <= self.shape[0]
            return Stand((last - first, 1), self, first)

        def reshape(self, shape):
            assert shape[0] * shape[1] == self.shape[0] * self.shape[1]
            return Stand(shape, self.slab, self.first)
    monkeypatch.setattr(cm, "empty", Stand)
    mats = cm.carve(shapes)
    assert [m.shape for m in mats] == shapes
    spans = sorted((id(m.slab), m.first, m.first + m.shape[0] * m.shape[1]) for m in mats)
    assert all(a[0] != b[0] or a[2] <= b[1] for a, b in zip(spans, spans[1:]))
