"""Build libmpx.so (the sm_100a engine behind include/mpx.h) in-tree with nvcc.

The kernel families compile in one file each (csrc/*.cu, see csrc/launch.h), in
parallel, into _build/ and link into one library next to this file, so that it
travels with the source tree; a file is compiled again when one of the headers
it includes has changed.  A second build of the same files with
-DMPX_BOUNDS_CHECK, libmpx_checked.so, verifies the index of every per-cell field
access (mpx_bounds_check reads the records).
"""
import concurrent.futures
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
UNITS = ["xthree", "xpass", "yz", "engine", "yzwarp", "yzlong", "yzthree", "thick", "pairs"]
CHECKED_UNITS = ["checked_" + u for u in UNITS]  # objects of the same files with the check
OUT = os.path.join(HERE, "libmpx.so")
OUT_CHECKED = os.path.join(HERE, "libmpx_checked.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr", "-Xfatbin", "-compress-all",
]


def nvcc_path():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _obj(unit):
    return os.path.join(OBJ, unit + ".o")


def _src(unit):
    return os.path.join(CSRC, unit.removeprefix("checked_") + ".cu")


def _deps(unit):
    """Files of this tree the unit was compiled from (the compiler's dependency file), or None
    where that file is missing or names another tree's (a copied _build folder)."""
    try:
        with open(os.path.join(OBJ, unit + ".d")) as f:
            words = f.read().replace("\\\n", " ").split()
    except OSError:
        return None
    deps = [w for w in words[1:] if w.startswith(ROOT + os.sep)]
    return deps if _src(unit) in deps else None


def _stale(unit):
    deps = _deps(unit)
    if deps is None or not os.path.exists(_obj(unit)):
        return True
    t = os.path.getmtime(_obj(unit))
    return any(not os.path.exists(d) or os.path.getmtime(d) > t for d in deps + [os.path.abspath(__file__)])


def up_to_date(out=OUT):
    units = CHECKED_UNITS if out == OUT_CHECKED else UNITS
    if not os.path.exists(out) or any(_stale(u) for u in units):
        return False
    return all(os.path.getmtime(_obj(u)) <= os.path.getmtime(out) for u in units)


def _run(cmd, verbose):
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + r.stdout)
    if verbose and r.stdout:
        print(r.stdout, file=sys.stderr)


def _command(out, extra=(), unit="engine"):
    """The nvcc command of `unit` into `out`; the checked library's adds the check."""
    checked = out == OUT_CHECKED or unit.startswith("checked_")
    return ([nvcc_path()] + NVCC_FLAGS + (["-DMPX_BOUNDS_CHECK"] if checked else []) + list(extra)
            + ["-I", os.path.join(ROOT, "include"), _src(unit), "-o", out])


def _compile(unit, extra, verbose):
    extra = list(extra) + ["-c", "-MMD", "-MF", os.path.join(OBJ, unit + ".d")]
    _run(_command(_obj(unit), extra, unit), verbose)


def build(force=False, verbose=False, extra=(), checked=True):
    """Compile libmpx.so (and libmpx_checked.so when `checked`) for sm_100a;
    returns the path of libmpx.so."""
    os.makedirs(OBJ, exist_ok=True)
    outs = [o for o in ([OUT, OUT_CHECKED] if checked else [OUT]) if force or not up_to_date(o)]
    units = [u for o in outs for u in (CHECKED_UNITS if o == OUT_CHECKED else UNITS) if force or _stale(u)]
    units.sort(key=lambda u: UNITS.index(u.removeprefix("checked_")))  # the longest first
    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, os.cpu_count() or 1)) as pool:
        for f in [pool.submit(_compile, u, extra, verbose) for u in units]:
            f.result()
    for out in outs:
        objs = [_obj(u) for u in (CHECKED_UNITS if out == OUT_CHECKED else UNITS)]
        _run([nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", out] + objs, verbose)
    return OUT


if __name__ == "__main__":
    force = "--force" in sys.argv
    extra = ["-Xptxas", "-v"] if "--ptxas" in sys.argv else []
    print(build(force=force or bool(extra), verbose=True, extra=extra, checked="--unchecked" not in sys.argv))
