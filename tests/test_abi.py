"""The C ABI library loads on a CPU-only machine, exports every function include/*.h
declares, checks its inputs on the host, and fails loudly (no CPU fallback) without a GPU."""
import ctypes as C
import glob
import os
import re

import numpy as np
import pytest

import dmplex_b200 as d
from dmplex_b200 import _lib
from conftest import ROOT, gpu_available, tables, trisk_grid


def declared_functions():
    names = set()
    for header in glob.glob(os.path.join(ROOT, "include", "*.h")):
        text = open(header).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        names |= set(re.findall(r"\b(trisk_\w+)\s*\(", text))
    return sorted(names)


def test_library_exports_every_declared_symbol():
    lib = C.CDLL(_lib.LIB_PATH)
    names = declared_functions()
    assert len(names) >= 30
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing


def test_struct_layouts_match():
    for which, cls in enumerate((_lib.TriskGrid, _lib.TriskCoefficients, _lib.TriskConfig, _lib.TriskPlex)):
        assert _lib.lib.trisk_struct_size(which) == C.sizeof(cls)
    from oracle.oracle import OracleModelStruct
    assert C.sizeof(OracleModelStruct) == C.sizeof(_lib.TriskCoefficients)


def test_bad_tables_are_rejected_on_the_host():
    t = dict(tables(3, "trisk", "cell"))
    bad = t["cell_edges"].copy()
    bad[4, 2] = t["ne"] + 7
    t["cell_edges"] = bad
    with pytest.raises(d.TriskError) as e:
        d.TRiSKShallowWater.from_coefficients(t, pv_flux="trisk", kinetic_energy="cell")
    assert e.value.status == 2 and "cell_edges" in str(e.value)
    t = dict(tables(3, "gassmann", "cell"))
    t["g_edges"] = None
    with pytest.raises(d.TriskError) as e:
        d.TRiSKShallowWater.from_coefficients(t, pv_flux="gassmann", kinetic_energy="cell")
    assert e.value.status == 1


def test_bad_arguments():
    with pytest.raises(ValueError):
        d.TRiSKShallowWater(trisk_grid(2), pv_flux="upwind")
    with pytest.raises(ValueError):
        d.TRiSKShallowWater(trisk_grid(2), kinetic_energy="edge")
    with pytest.raises(d.TriskError) as e:
        d.create_hexagon_mesh(-1)
    assert e.value.status == 1


def test_no_gpu_fails_loudly():
    if gpu_available():
        pytest.skip("a GPU is present")
    with pytest.raises(d.TriskError) as e:
        d.TRiSKShallowWater(trisk_grid(2))
    assert e.value.status == 3


def test_last_error_is_thread_local_and_bounded():
    with pytest.raises(d.TriskError):
        d.create_hexagon_mesh(11)
    buf = C.create_string_buffer(8)
    n = _lib.lib.trisk_last_error(buf, len(buf))
    assert n > 7 and len(buf.value) == 7


def test_tables_are_deterministic():
    """The host table builder gives identical arrays on every call (the parity fixtures
    depend on it)."""
    a = d.model_tables(d.TRiSKGrid(d.create_hexagon_mesh(4, centroidal=True)), pv_flux="gassmann",
                       kinetic_energy="mixed")
    b = d.model_tables(d.TRiSKGrid(d.create_hexagon_mesh(4, centroidal=True)), pv_flux="gassmann",
                       kinetic_energy="mixed")
    for k, v in a.items():
        if isinstance(v, np.ndarray):
            assert np.array_equal(v, b[k]), k


def test_which_pointers_a_kernel_may_access(tmp_path):
    """csrc/pointers.hpp, compiled alone: aligned memory of the model's device and aligned managed
    memory of any; another device's memory and other byte addresses are left to the copy engine."""
    import subprocess
    source = tmp_path / "rule.cpp"
    source.write_text("""
#include <cstdio>
#include "pointers.hpp"
int main() {
  for (long address = 4096; address <= 4100; address += 4)
    for (int managed = 0; managed < 2; ++managed)
      for (int device = 0; device < 2; ++device)
        std::putchar('0' + trisk::kernel_can_access(reinterpret_cast<void*>(address), managed, device, 0));
}
""")
    exe = str(tmp_path / "rule")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "dmplex_b200", "csrc"),
                    str(source), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out == "1011" + "0000"  # [own, other] device memory, then managed; unaligned: never
