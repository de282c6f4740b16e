"""Builds the Tier-1 kernels' device code for the CPU warp emulator
(cuda_runtime.h here): a kernel file up to its launchers, with its two inline
PTX instructions written out, compiled by g++ with the driver in drivers.cc."""
import ctypes as C
import re
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent.parent
CSRC = ROOT / "thousandthchicken_b200" / "csrc"

# kernel file, the line that its device part ends before
PARTS = {"EMU_WARP": ("t1_decode_warp.cu", "// The blocks of a launch"),
         "EMU_GROUPS": ("t1_decode.cu", "// Persistent Tier-1 launch over one magnitude class."),
         "EMU_ENCODE": ("t1_encode.cu", "}  // namespace\n\ncudaError_t launch_t1_encode")}


def _cut(text, before):
    assert text.count(before) == 1, before
    return text[:text.index(before)]


def build(kind, outdir: Path, source: Path | None = None) -> C.CDLL:
    """The emulated kernels of PARTS[kind], as a loaded library."""
    name, end = PARTS[kind]
    text = _cut((source or CSRC / name).read_text(), end)
    internal = (CSRC / "tc_internal.cuh").read_text()
    consts = "\n".join(re.findall(r"^#define TC_DERR_.*$", internal, re.M)) + "\nnamespace tc {\n" + \
        re.search(r"constexpr int kStyleDecodeBits[^;]*;", internal).group(0) + "\n}\n"
    assert '#include "tc_internal.cuh"' in text
    text = text.replace('#include "tc_internal.cuh"', '#include "tc_j2k.h"\n' + consts)
    text = re.sub(r'asm\("bfind\.u32 [^;]*;"[^;]*;', "r = x ? 31 - __builtin_clz(x) : -1;", text)
    text = re.sub(r'asm\("bfind\.shiftamt\.u32 [^;]*;"[^;]*;', "r = x ? __builtin_clz(x) : -1;", text)
    assert "asm(" not in text
    src, so = outdir / f"{kind.lower()}.inc", outdir / f"{kind.lower()}.so"
    src.write_text(text)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-w", f"-I{HERE}", f"-I{CSRC}", f"-I{ROOT / 'include'}",
                    f"-D{kind}", f'-DEMU_SOURCE="{src}"', str(HERE / "drivers.cc"), "-o", str(so)], check=True)
    return C.CDLL(str(so))
