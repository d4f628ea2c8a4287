"""A z-kernel tile whose copy does not arrive in time (the bounded wait of its
barrier runs out) leaves NaN in its results in every form of the kernel, so that
a caller sees it: built for the host with a TMA that never completes."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "bigdft-suite_b200" / "csrc"

NEVER = """#pragma once
#include <cuda.h>
#include <stdint.h>
namespace wvlh {
inline unsigned smem_addr(const void *) { return 0; }
inline void mbar_init(uint64_t *, unsigned) {}
inline void mbar_expect_tx(uint64_t *, unsigned) {}
inline bool mbar_wait_bounded(uint64_t *, unsigned) { return false; }
inline void tma_load_4d(void *, const CUtensorMap *, int, int, int, int, uint64_t *) {}
}
"""


@pytest.fixture(scope="module")
def timed_out(tmp_path_factory):
    cuda = Path("/usr/local/cuda/include")
    if not cuda.exists():
        pytest.skip("no CUDA headers")
    tmp = tmp_path_factory.mktemp("ztile")
    text = (CSRC / "wvlh_fused_impl.cuh").read_text()
    cut = text.index("// host launchers")
    (tmp / "ztile.cuh").write_text(text[:cut] + "\n}  // namespace wvlh\n")
    (tmp / "wvlh_tma.cuh").write_text(NEVER)
    so = tmp / "ztile.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w", "-I", str(tmp), "-I", str(cuda), "-I",
                    str(CSRC), str(HERE / "native" / "ztile_host.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so)).ztile_timed_out


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("chain", [0, 1, 2])
@pytest.mark.parametrize("n,tile", [((3, 2, 2), 0), ((9, 8, 5), 1), ((20, 3, 9), 2), ((20, 3, 9), 5)])
def test_timed_out_tile_is_nan(timed_out, prec, chain, n, tile):
    assert timed_out(prec, chain, *n, tile) == 0
