"""In-tree build of librewy_b200.so (sm_100a, nvcc) and of the torch operators over it (rewy_b200_torch.so, g++).
``python -m rewy_b200.build``."""
import hashlib
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from importlib.metadata import version
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "csrc" / "build"
LIB = PKG / "librewy_b200.so"
TORCH_LIB = PKG / "rewy_b200_torch.so"
SOURCES = ("capi.cu", "prepare.cu", "prepare_tc.cu", "state_scan.cu", "state_scan_tc.cu", "state_scan_split.cu", "chunk_adjoint.cu", "chunk_adjoint_tc.cu", "tc_selftest.cu", "wrappers.cu", "rows.cu", "chunk_fwd.cu", "chunk_fwd_tc.cu", "chunk_output_tc.cu")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--expt-relaxed-constexpr", "--expt-extended-lambda", "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


def _digest(paths):
    h = hashlib.sha256()
    for p in sorted(paths):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    h.update(version("torch").encode())   # the torch operators are compiled against its headers
    return h.hexdigest()


def _build_torch_library():
    """csrc/binding.cpp against the headers of the installed torch, linked to librewy_b200.so beside it."""
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", str(CSRC / "binding.cpp"), "-o", str(TORCH_LIB),
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-isystem{p}" for p in (root / "include", root / "include/torch/csrc/api/include", cuda / "include")),
           f"-L{root / 'lib'}", f"-L{PKG}", "-l:librewy_b200.so", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
           "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"the torch operator library did not build:\n{r.stderr[-6000:]}")


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ for sm_100a and link the shared library.  Returns its path."""
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [CSRC / "binding.cpp"] + [PKG.parent / "include" / "rewy_b200.h"]
    stamp = OBJ / "stamp.txt"
    digest = _digest(deps)
    if not force and LIB.exists() and TORCH_LIB.exists() and stamp.exists() and stamp.read_text() == digest:
        return LIB
    OBJ.mkdir(parents=True, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src):
        obj = OBJ / (src[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(CSRC / src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        (OBJ / (src[:-3] + ".ptxas.txt")).write_text(r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stderr[-6000:]}")
        if verbose:
            print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr[-4000:]}")
    _build_torch_library()
    stamp.write_text(digest)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
