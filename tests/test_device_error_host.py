"""The message of PIBEM_ETIMEDOUT names the kernels whose bounded wait gave up (pibem_internal.h)."""
import ctypes as C
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_message_by_source(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(f'#include "{REPO}/pi-bem_gb300/csrc/pibem_internal.h"\n'
                   "using namespace pibem;\n"
                   'extern "C" const char *text(int ilu, int tr) {\n'
                   "  return device_error_text((ilu ? DEV_TIMEOUT_ILU : 0) | (tr ? DEV_TIMEOUT_TRANSLATIONS : 0)); }\n")
    out = tmp_path / "t.so"
    subprocess.run(["g++", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include", "-o", str(out), str(src)],
                   check=True)
    lib = C.CDLL(str(out))
    lib.text.restype = C.c_char_p
    ilu, tr, both = (lib.text(*a).decode() for a in ((1, 0), (0, 1), (1, 1)))
    assert "ILU" in ilu and "translations" not in ilu
    assert "translations" in tr and "ILU" not in tr
    assert "ILU" in both and "translations" in both
