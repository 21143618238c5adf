"""CPU checks of the drop-in boundary: the C-ABI library loads without a GPU, exports every symbol the header
declares, and its host-only entry points (generators, argument validation) behave."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "et_b200.h")


@pytest.fixture(scope="module")
def lib():
    import et_b200
    from et_b200 import build
    build.build()                      # no-op when the in-tree library is current
    return et_b200.lib()


def declared_symbols():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(et_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported(lib):
    names = declared_symbols()
    assert len(names) >= 30
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, f"declared in include/et_b200.h but not exported: {missing}"


def test_every_declaration_cites_the_reference_or_says_it_has_no_counterpart():
    text = open(HEADER).read()
    for name in declared_symbols():
        idx = text.index(name + "(")
        before = text[:idx]
        comment = before[before.rfind("/*"):]
        block_start = text.rfind("/* ----", 0, idx)
        section = text[block_start:idx] if block_start >= 0 else comment
        assert re.search(r"\.(h|cu):\d+|no counterpart|et_last_error|et_version", section + name), name


def test_version_and_error_text(lib):
    assert lib.et_version() == 100
    rc = lib.et_skip_layernorm(None, None, None, None, 4, 768, None)
    assert rc == 1                                      # ET_ERR_INVALID before any CUDA call
    assert b"null pointer" in lib.et_last_error()


def test_generators_match_oracle_without_gpu(lib, orc):
    import et_b200 as et
    for (nrow, ncol, s, seed, bern) in [(768, 768, 0.5, 1, False), (768, 3072, 0.75, 3, True), (64, 64, 1.0, 6, False)]:
        rp, ro = et.gen_sparse_tile_mat(nrow, ncol, s, seed, bern)
        rp2, ro2 = orc.gen_sparse_tile_mat(nrow, ncol, s, seed, bern)
        assert (rp == rp2).all() and (ro == ro2).all()
    a = et.gen_sparse_row_mat(768, 0.5, 9, 12)
    assert (a == orc.gen_sparse_row_mat(768, 0.5, 9, 12)).all()
    assert (et.build_head_ptr(a, 12, 768) == orc.head_ptr(a, 12, 768)).all()


def test_generator_argument_checks(lib):
    import et_b200 as et
    with pytest.raises(et.EtError):
        et.gen_sparse_tile_mat(100, 64, 0.5, 1)          # not a multiple of 16
    with pytest.raises(et.EtError):
        et.gen_sparse_tile_mat(64, 64, 1.5, 1)           # sparsity outside [0, 1]
    with pytest.raises(et.EtError):
        et.build_head_ptr(np.array([5, 3], dtype=np.int32), 2, 64)   # not ascending


def test_lengths_may_be_any_numbers_that_numpy_makes_ints_of(lib):
    """Ints of any kind, numpy scalars and whole floats, in lists, tuples and arrays."""
    import ctypes
    from et_b200.ops import _ints
    for values in ([3, 5], (3, 5), [3.0, 5.0], [np.float32(3), 5], [np.int64(3), np.int32(5)], np.array([3, 5]), np.array([3.0, 5.0])):
        address, count, owner = _ints(values)
        assert count == 2 and list((ctypes.c_int * 2).from_address(address)) == [3, 5], (values, owner)


def test_tile_weight_validation_happens_before_any_device_work(lib):
    import et_b200 as et
    data = np.zeros((2, 256), dtype=np.float16)
    with pytest.raises(et.EtError) as e:
        et.TileWeight(64, 32, 128, data, np.array([0, 1, 2], dtype=np.int32), np.array([8, 16], dtype=np.int32))
    assert e.value.code == 1


def test_shim_headers_compile_standalone(tmp_path):
    """The headers with the reference's names are self-contained (host compile only, no GPU)."""
    src = tmp_path / "t.cu"
    src.write_text('#include <encoder/encoder.h>\n#include <test/utils.h>\n'
                   'int probe(int d) { return (int)Encoder_length::buffer_size(d, 128, 12) + Encoder_base::buffer_num; }\n')
    res = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-c",
                          "-I", os.path.join(ROOT, "include"), str(src), "-o", str(tmp_path / "t.o")],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr


def test_product_does_not_import_the_oracle():
    for base, _, files in os.walk(os.path.join(ROOT, "et_b200")):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h")):
                text = open(os.path.join(base, f)).read()
                assert "oracle" not in text.lower() or f == "build.py", f
