"""The C-ABI library loads without a GPU and exports every symbol include/xattn_b200.h declares."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from xattn_b200 import _lib, build
    build.build()
    return _lib.load()


def _declared():
    text = open(os.path.join(ROOT, "include", "xattn_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(xattn_b200_\w+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound(lib):
    from xattn_b200 import _lib
    names = _declared()
    assert len(names) >= 10
    for n in names:
        assert hasattr(lib, n), f"{n} declared in the header but not exported"
    assert sorted(_lib.SIGNATURES) == names


def test_host_only_entry_points(lib):
    assert lib.xattn_b200_version() >= 100
    assert lib.xattn_b200_error_string(0) == b"ok"
    assert b"argument" in lib.xattn_b200_error_string(1)
    for L, want in ((1000, 2048), (4096, 4096), (16384, 16384), (32768, 8192), (62208, 4096), (131072, 2048)):
        assert lib.xattn_b200_default_chunk_size(L) == want      # Xattention.py:322-331
    out = (ctypes.c_int * 8)()
    assert lib.xattn_b200_estimate_geometry(1024, 5000, 2048, 16, 128, out) == 0
    assert list(out) == [2048, 6144, 16, 48, 1, 3, 16, 32]
    assert lib.xattn_b200_estimate_geometry(5000, 1024, 2048, 16, 128, out) != 0   # k chunks < q chunks
    assert lib.xattn_b200_estimate_workspace_bytes(1, 32, 131072, 131072, 16, 128, 2048) > (1 << 30)
    assert lib.xattn_b200_estimate_workspace_bytes(1, 32, 4096, 4096, 3, 128, 2048) == 0       # bad stride


def test_workspace_bytes_cover_every_mask_and_semantics(lib):
    for stride in (4, 8, 16, 32):
        for chunk in (128, 256, 384, 640, 1024, 1152, 2048, 4096):
            for nq, extra, ragged in ((1, 0, 0), (1, 1, 0), (2, 0, 5), (3, 0, 0), (3, 2, 100), (8, 0, 0)):
                q, k = nq * chunk - ragged, (nq + extra) * chunk - ragged
                most = lib.xattn_b200_estimate_workspace_bytes(1, 8, q, k, stride, 128, chunk)
                for causal, semantics in ((0, 0), (0, 1), (1, 0), (1, 1), (1, 2)):
                    need = lib.xattn_b200_estimate_workspace_bytes_ex(1, 8, q, k, stride, 128, chunk, causal, semantics)
                    assert need <= most, (stride, chunk, q, k, causal, semantics)


def test_ops_refuse_cpu_tensors():
    import torch
    from xattn_b200 import Xattention_prefill
    from xattn_b200._lib import XattnB200Error
    q = torch.zeros(1, 1, 128, 128, dtype=torch.bfloat16)
    with pytest.raises(XattnB200Error):
        Xattention_prefill(q, q, q, stride=16)


def test_reference_import_path():
    from xattn.src.Xattention import Xattention_prefill, xattn_estimate  # noqa: F401
    from xattn.src.utils import find_blocks_chunked  # noqa: F401


def test_the_arguments_of_the_combined_call_are_bound_in_order():
    from xattn_b200 import _lib
    text = open(os.path.join(ROOT, "include", "xattn_b200.h")).read()
    body = re.search(r"typedef struct \{([^}]*)\} xattn_b200_estimate_select_args;", text).group(1)
    kinds = {"int": ctypes.c_int, "int64_t": ctypes.c_int64, "float": ctypes.c_float, "double": ctypes.c_double, "size_t": ctypes.c_size_t}
    fields = []
    for line in body.split(";"):
        words = line.replace("const ", "").split(None, 1)
        if words:
            fields += [(n.strip(" *"), ctypes.c_void_p if "*" in n else kinds[words[0].strip("*")])
                       for n in (words[1] if "*" not in words[0] else "*" + words[1]).split(",")]
    assert fields == _lib.EstimateSelectArgs._fields_
