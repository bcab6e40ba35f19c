import ctypes
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

GOLDEN = Path(__file__).resolve().parent / "golden"


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


def load_golden(name: str) -> dict:
    """Golden fixtures as torch tensors; bf16-exact inputs (stored as their upper 16 bits) come back as fp32."""
    out = {}
    with np.load(GOLDEN / name) as z:
        for k in z.files:
            a = z[k]
            if a.dtype == np.uint16:
                a = (a.astype(np.uint32) << 16).view(np.float32)
            out[k] = torch.from_numpy(np.ascontiguousarray(a))
    return out


@pytest.fixture(scope="session")
def golden_attention():
    return load_golden("attention_ref.npz")


@pytest.fixture(scope="session")
def golden_indices():
    return load_golden("indices_ref.npz")


@pytest.fixture(scope="session")
def golden_csla():
    return load_golden("csla_ref.npz")


@pytest.fixture(scope="session")
def golden_scalekv():
    return load_golden("scalekv_ref.npz")


@pytest.fixture(scope="session")
def golden_prologue():
    return load_golden("prologue_ref.npz")


_ROWS_VIEW = """
#include "rows_view.cuh"
extern "C" int rows_view(int B, int H, int L, int D, long long sb, long long sh, long long sl, long long* out) {
  const lvar::RowsView r = lvar::rows_view(B, H, L, D, sb, sh, sl);
  out[0] = r.rb; out[1] = r.rh; out[2] = r.ch; out[3] = r.rows; out[4] = r.width;
  return r.ok ? 1 : 0;
}
"""


@pytest.fixture(scope="session")
def rows_view(tmp_path_factory):
    """The library's gather rule, compiled for the host: (shape, strides) -> (rb, rh, ch, rows, width), or None for the copies."""
    d = tmp_path_factory.mktemp("rows_view")
    (d / "rows_view.cpp").write_text(_ROWS_VIEW)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", str(ROOT / "lvar_b200" / "csrc"), "-o", str(d / "rows_view.so"),
                    str(d / "rows_view.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "rows_view.so")).rows_view
    fn.argtypes = [ctypes.c_int] * 4 + [ctypes.c_longlong] * 3 + [ctypes.POINTER(ctypes.c_longlong)]

    def call(shape, strides):
        out = (ctypes.c_longlong * 5)()
        return tuple(out) if fn(*shape, *strides[:3], out) else None
    return call
