"""Build libb200engine.so in-tree with nvcc for sm_100a (cross-compiles without a GPU).

The shared library is the product: a C-ABI engine (include/b200engine.h) with no Python or torch
dependency.  Python only loads it through ctypes (kubeai_b200/_lib.py).
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent
CSRC = ROOT / "csrc"
LIB = ROOT / "lib" / "libb200engine.so"
OBJ = ROOT / "lib" / "obj"
# The Python side's one native helper (csrc/pyfeed.cc).  It reads lists, tuples and arrays by the layouts of one interpreter, so its name says which:
# another one does not find it and forms the entries with numpy.
FEED = ROOT / ("_feed" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))

SOURCES = [
    "gemm_tcgen05.cu",
    "gemm2_tcgen05.cu",
    "gemm3_tcgen05.cu",
    "gemm_grouped.cu",
    "chain_tcgen05.cu",
    "attention.cu",
    "attention_tc.cu",
    "elementwise.cu",
    "linear.cu",
    "linear_stream.cu",
    "linear_cluster.cu",
    "norm_act.cu",
    "gla.cu",
    "scan_chunk.cu",
    "scan_parallel.cu",
    "delta.cu",
    "delta_chunk.cu",
    "latent_attention.cu",
    "moe.cu",
    "hyper.cu",
    "window_attention.cu",
    "prompt_attention.cu",
    "ssm.cu",
    "nomanex.cu",
    "zinavik.cu",
    "mulenex.cu",
    "nagilix.cu",
    "soselix.cu",
    "dabodra.cu",
    "model_registry.cc",
    "abi_ops.cu",
    "engine.cu",
    "router.cc",
    "loader.cc",
    "tokenizer.cc",
    "server.cc",
    "harness.cc",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-Wall,-Wno-unused-function",
    "-diag-suppress", "177",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _feed_flags():
    """Include flags of the Python helper; none where Python's or numpy's headers are not installed (engine.py works without it)."""
    try:
        import numpy
    except ImportError:
        return []
    dirs = [sysconfig.get_paths()["include"], numpy.get_include(), str(ROOT.parent / "include")]
    if not os.path.exists(os.path.join(dirs[0], "Python.h")) or not os.path.isdir(dirs[1]):
        return []
    return [f for d in dirs for f in ("-I", d)]


def _digest(paths) -> str:
    h = hashlib.sha256()
    for p in sorted(paths):
        h.update(str(p).encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def _feed_digest(flags) -> str:
    """What the helper was made from: its source, the entry it fills, the interpreter and the numpy whose layouts it knows."""
    import numpy
    h = hashlib.sha256(_digest([CSRC / "pyfeed.cc", ROOT.parent / "include" / "b200engine.h"]).encode())
    h.update(" ".join([sys.version, numpy.__version__, *flags]).encode())
    return h.hexdigest()


def build_feed(force: bool = False) -> bool:
    """Build the Python helper where it can be built; whether it is there.  Without it engine.py forms the entries with numpy, so a
    compiler that fails is reported and no more."""
    plain = FEED.with_name("_feed.so")      # a name that every interpreter takes for its own
    if plain != FEED:
        plain.unlink(missing_ok=True)
    flags = _feed_flags()
    if not flags:
        return FEED.exists()
    stamp = OBJ / "feed_digest.txt"
    digest = _feed_digest(flags)
    if not force and FEED.exists() and stamp.exists() and stamp.read_text() == digest:
        return True
    OBJ.mkdir(parents=True, exist_ok=True)
    FEED.unlink(missing_ok=True)
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", *flags, str(CSRC / "pyfeed.cc"), "-o", str(FEED)]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        failed = f"{r.stdout}\n{r.stderr}" if r.returncode else ""
    except OSError as e:
        failed = str(e)
    if failed:
        print(f"kubeai_b200: building {FEED.name} failed, entries will be formed by numpy:\n{failed}", file=sys.stderr)
        return False
    stamp.write_text(digest)
    return True


def build(force: bool = False, verbose: bool = False) -> Path:
    build_feed(force)
    srcs = [CSRC / s for s in SOURCES if (CSRC / s).exists()]
    deps = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + [ROOT.parent / "include" / "b200engine.h"] + list((ROOT.parent / "cmd").glob("*.cc"))
    stamp = OBJ / "digest.txt"
    digest = _digest(srcs + deps)
    if not force and LIB.exists() and stamp.exists() and stamp.read_text() == digest:
        return LIB
    OBJ.mkdir(parents=True, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: Path) -> Path:
        obj = OBJ / (src.name + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-x", "cu", "-c", str(src), "-o", str(obj)]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart", "-lpthread", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    # the two process entry points (cmd/): server and load generator, linked against the library
    bindir = ROOT / "bin"
    bindir.mkdir(exist_ok=True)
    for name in ("b200serve", "b200bench"):
        src = ROOT.parent / "cmd" / f"{name}.cc"
        if not src.exists():
            continue
        cmd = [nvcc, "-O2", "-std=c++17", "-x", "cu", str(src), "-o", str(bindir / name), "-L", str(LIB.parent),
               "-lb200engine", "-Xlinker", "-rpath", "-Xlinker", "$ORIGIN/../lib", "-lcudart", "-lpthread"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"building {name} failed:\n{r.stdout}\n{r.stderr}")
    stamp.write_text(digest)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
