"""In-tree build of libmccl.so (host C++ with g++, device code with nvcc for sm_100a) and of the torch binding.

`python -m mccl_b200._build` compiles every file under csrc/ that changed since its object was made, or whose headers did, and links
mccl_b200/lib/libmccl.so, and from csrc/torch the torch binding, one file per torch version (its C++ interface is no other's).  Objects
live in build/ (ignored by git); the shared libraries stay inside the package so that they travel with the source tree.
"""
from __future__ import annotations

import concurrent.futures as cf
import fcntl
import os
import shutil
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "csrc"
OBJ = ROOT / "build" / "obj"
TORCH_SRC = CSRC / "torch"                       # the torch binding: a library of its own, so that libmccl needs no torch
LIB = ROOT / "mccl_b200" / "lib" / "libmccl.so"
CUDA_HOME = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
NVCC = str(CUDA_HOME / "bin" / "nvcc")

CXXFLAGS = ["-O2", "-g1", "-fPIC", "-std=c++17", "-Wall", "-Wextra", "-Wno-unused-parameter", "-pthread",
            f"-I{ROOT / 'include'}", f"-I{CSRC}", f"-I{CUDA_HOME / 'include'}"]
NVCCFLAGS = ["-O3", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
             "-Xcompiler", "-fPIC,-Wall,-Wno-unused-parameter", f"-I{ROOT / 'include'}", f"-I{CSRC}",
             "--expt-relaxed-constexpr", "-Xptxas", "-v"]


def _stale(src: Path, obj: Path) -> bool:
    """Whether `src` or a file it included when `obj` was made is newer than `obj`."""
    dep = obj.with_suffix(".d")
    if not obj.exists() or not dep.exists():
        return True
    made = obj.stat().st_mtime
    for name in dep.read_text().replace("\\\n", " ").split(":", 1)[1].split():
        f = Path(name)
        if not f.exists() or f.stat().st_mtime > made:
            return True
    return False


def _compile(src: Path, obj: Path, extra: list[str]) -> tuple[Path, str]:
    obj.parent.mkdir(parents=True, exist_ok=True)
    if src.suffix == ".cu":
        cmd = [NVCC, *NVCCFLAGS, "-MMD", "-MF", str(obj.with_suffix(".d")), "-c", str(src), "-o", str(obj)]
    else:
        cmd = ["g++", *CXXFLAGS, *extra, "-MMD", "-MF", str(obj.with_suffix(".d")), "-c", str(src), "-o", str(obj)]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        raise RuntimeError(f"compile failed: {' '.join(cmd)}\n{p.stdout}\n{p.stderr}")
    log = p.stderr if src.suffix == ".cu" else ""
    if src.suffix == ".cu":
        (obj.with_suffix(".ptxas.txt")).write_text(p.stderr)
    return src, log


def _torch_tag(version: str) -> str:
    return "".join(c if c.isalnum() or c in ".-" else "_" for c in version)


def ext_path(version: str) -> Path:
    """The binding's file for this version of torch."""
    return LIB.with_name(f"mccl_torch-{_torch_tag(version)}.so")


def _torch_flags() -> tuple[list[str], list[str]] | None:
    """Compile and link flags of the torch binding; None where torch is not installed or has no CUDA (the tcp transport and
    numpy arrays work without)."""
    import sysconfig
    try:
        import torch
    except ImportError:
        return None
    if torch.version.cuda is None:
        return None
    inc = Path(torch.__file__).parent / "include"
    lib = Path(torch.__file__).parent / "lib"
    cflags = [f"-isystem{inc}", f"-isystem{inc / 'torch/csrc/api/include'}", f"-isystem{sysconfig.get_paths()['include']}",
              "-DTORCH_EXTENSION_NAME=mccl_torch", "-DTORCH_API_INCLUDE_EXTENSION_H",
              f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-fvisibility=hidden"]
    lflags = [f"-L{lib}", "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", f"-L{LIB.parent}", "-lmccl",
              "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{lib}"]
    return cflags, lflags


def _link(cmd: list[str], target: Path) -> None:
    # Linked beside the target and renamed into place: whoever copies or loads the tree never sees half a library.
    target.parent.mkdir(parents=True, exist_ok=True)
    tmp = target.with_name(f".{target.name}.{os.getpid()}.tmp")
    p = subprocess.run([*cmd, "-o", str(tmp)], capture_output=True, text=True)
    if p.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f"link failed: {' '.join(cmd)}\n{p.stdout}\n{p.stderr}")
    os.replace(tmp, target)


def build(verbose: bool = False, force: bool = False) -> Path:
    if shutil.which(NVCC) is None and not Path(NVCC).exists():
        raise RuntimeError(f"nvcc not found at {NVCC}")
    OBJ.mkdir(parents=True, exist_ok=True)
    with open(OBJ.parent / "lock", "w") as lock:         # ranks that find a library missing build it once
        fcntl.flock(lock, fcntl.LOCK_EX)
        return _build_locked(verbose, force)


def _build_locked(verbose: bool, force: bool) -> Path:
    srcs = sorted(list(CSRC.rglob("*.cc")) + list(CSRC.rglob("*.cu")))
    torch_flags = _torch_flags()
    if torch_flags is not None:
        import torch
        ext = ext_path(torch.__version__)
    jobs, objs, ext_objs = [], [], []
    for s in srcs:
        in_ext = TORCH_SRC in s.parents
        if in_ext and torch_flags is None:
            continue
        o = OBJ / s.relative_to(CSRC).with_suffix(s.suffix + ".o")
        if in_ext:
            o = OBJ / ext.stem / o.name
        (ext_objs if in_ext else objs).append(o)
        if force or _stale(s, o):
            jobs.append((s, o, torch_flags[0] if in_ext else []))
    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 4)) as ex:
            for src, log in ex.map(lambda job: _compile(*job), jobs):
                if verbose:
                    print(f"[mccl build] {src.relative_to(ROOT)}")
                    if log:
                        print(log)
    if jobs or not LIB.exists():
        _link([NVCC, "-shared", *map(str, objs), "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xlinker", "--no-undefined", "-lpthread", "-ldl", "-lrt"], LIB)
        if verbose:
            print(f"[mccl build] linked {LIB.relative_to(ROOT)}")
    if ext_objs and (jobs or not ext.exists()):
        _link(["g++", "-shared", *map(str, ext_objs), *torch_flags[1]], ext)
        if verbose:
            print(f"[mccl build] linked {ext.relative_to(ROOT)}")
    return LIB


def resources() -> str:
    """Markdown table of what ptxas reported for every kernel of the last build (registers, spills, static shared
    memory), template instantiations of one kernel folded into one row."""
    import re
    from collections import OrderedDict
    found = []
    for f in sorted(OBJ.rglob("*.ptxas.txt")):
        entry, spill = None, ("0", "0", "0")
        for line in f.read_text().splitlines():
            m = re.search(r"Compiling entry function '(\S+)' for 'sm_100a'", line)
            if m:
                entry, spill = m.group(1), ("0", "0", "0")
                continue
            m = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", line)
            if m and entry:
                spill = m.groups()
            m = re.search(r"Used (\d+) registers", line)
            if m and entry:
                smem = re.search(r"(\d+) bytes smem", line)
                found.append((f.name.replace(".ptxas.txt", ""), entry, int(m.group(1)),
                              int(spill[1]) + int(spill[2]), int(smem.group(1)) if smem else 0))
                entry = None
    names = subprocess.run(["c++filt"], input="\n".join(k[1] for k in found), capture_output=True,
                           text=True).stdout.splitlines()
    rows: "OrderedDict[tuple, list]" = OrderedDict()
    for k, name in zip(found, names):
        name = name.replace("(anonymous namespace)::", "").replace("mccl::", "")
        name = re.sub(r"^void ", "", re.sub(r"\(.*\)$", "", name))
        base = name.split("<")[0]
        rows.setdefault((k[0], base), []).append(k)
    out = ["| file | kernel | instantiations | registers | spill bytes (stores + loads), worst | static smem bytes, worst |",
           "|---|---|---|---|---|---|"]
    for (src, base), ks in rows.items():
        regs = [k[2] for k in ks]
        out.append(f"| {src} | `{base}` | {len(ks)} | {min(regs)}" + (f" - {max(regs)}" if max(regs) != min(regs) else "")
                   + f" | {max(k[3] for k in ks)} | {max(k[4] for k in ks)} |")
    out.append("")
    out.append(f"{len(found)} kernels in {len(rows)} families; {sum(1 for k in found if k[3])} with spills.")
    return "\n".join(out)


if __name__ == "__main__":
    if "--resources" in sys.argv:
        print(resources())
    else:
        build(verbose=True, force="--force" in sys.argv)
