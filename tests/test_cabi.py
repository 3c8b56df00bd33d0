"""The C ABI: the shared library loads without a GPU and exports every symbol that
include/bamboo_b200.h declares; the Python binding mirrors the descriptor struct."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "bamboo_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(bb_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from bamboo_b200 import lib
    handle = lib.load()
    names = declared_symbols()
    assert len(names) >= 18
    for name in names:
        assert hasattr(handle, name), name
    assert handle.bb_version() >= 100


def test_gemm_descriptor_layout_matches_header():
    from bamboo_b200 import lib
    text = open(os.path.join(ROOT, "include", "bamboo_b200.h")).read()
    body = text[text.index("typedef struct bb_gemm_desc"):text.index("} bb_gemm_desc;")]
    body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
    fields = re.findall(r"(?:const\s+)?(?:void\*|long long|int)\s+([A-Za-z0-9_, ]+);", body)
    flat = [f.strip() for group in fields for f in group.split(",")]
    assert flat == [name for name, _ in lib.GemmDesc._fields_]
    assert ctypes.sizeof(lib.GemmDesc) % 8 == 0


def test_argument_errors_do_not_need_a_gpu():
    from bamboo_b200 import lib
    handle = lib.load()
    rc = handle.bb_gemm_bf16(None, None)
    assert rc == -1 and b"bb_gemm_bf16" in handle.bb_last_error()


@pytest.mark.parametrize("tile_n", [64, 96, 512, -1])
@pytest.mark.parametrize("split_k", [0, 1, 4])
def test_a_tile_that_does_not_exist_is_refused_with_and_without_a_split(tile_n, split_k):
    from bamboo_b200 import lib
    handle, fake = lib.load(), 1 << 20
    d = lib.GemmDesc(M=128, N=128, K=1024, A=fake, lda=1024, B=fake, ldb=1024, D=fake, ldd=128, tile_n=tile_n, split_k=split_k)
    assert handle.bb_gemm_bf16(ctypes.byref(d), None) == -1
    assert b"tile_n" in handle.bb_last_error()
