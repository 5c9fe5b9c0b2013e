"""The C ABI library loads and exports every symbol include/*.h declares
(no compute calls: these run without a GPU)."""
import ctypes
import glob
import os
import re
import subprocess

import numpy as np

from conftest import ROOT, golden

import nbody_gb300 as nb
from nbody_gb300 import _lib


def declared_symbols():
    names = set()
    for h in glob.glob(os.path.join(ROOT, "include", "*.h")):
        text = open(h).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        for m in re.finditer(r"NBGB_API\s+[\w\s\*]+?\b(\w+)\s*\(", text):
            names.add(m.group(1))
    return names


def test_header_declares_the_drop_in_signature():
    names = declared_symbols()
    assert "ComputeGravitation_GPU_GB300" in names
    text = open(os.path.join(ROOT, "include", "nbody_gb300.h")).read()
    # the reference's pfnComputeGravitation_AOS_t (src/nbody.h:68)
    assert re.search(r"float\s+ComputeGravitation_GPU_GB300\(float \*force, float \*posMass, "
                     r"float softeningSquared,\s+size_t N\)", text)


def test_library_exports_every_declared_symbol():
    lib = ctypes.CDLL(_lib.LIB_PATH)
    names = declared_symbols()
    assert len(names) >= 30
    missing = [n for n in sorted(names) if not hasattr(lib, n)]
    assert not missing, missing


def test_exports_are_c_linkage_and_nothing_else_leaks():
    out = subprocess.run(["nm", "-D", "--defined-only", _lib.LIB_PATH], capture_output=True,
                         text=True, check=True).stdout
    exported = {line.split()[-1] for line in out.splitlines() if " T " in line}
    assert declared_symbols() == exported


def test_python_binding_covers_the_header():
    assert declared_symbols() == set(_lib.SIGNATURES)


def test_version_and_status_strings():
    assert b"sm_103a" in _lib.load().nbgb_version()
    assert _lib.load().nbgb_status_string(0) == b"ok"
    assert b"workspace" in _lib.load().nbgb_status_string(-2)


def test_library_is_built_for_sm_103a_only():
    import nbody_gb300.build as B
    assert B.ARCH == ["-gencode", "arch=compute_103a,code=sm_103a"]


def test_host_ic_reference_matches_reference_bodies():
    g = golden("refic1024_seed7")
    pm, vm = nb.ic_reference(1024, 7)
    assert np.array_equal(pm, g["posMass"]) and np.array_equal(vm, g["velInvMass"])


def test_host_crosscheck_metric_matches_oracle():
    from oracle import oracle as O
    g = golden("ball2048")
    f = O.ieee().forces_aos(g["posMass"], float(g["eps2"]))
    assert nb.crosscheck_max_rel_error(f, g["force_aos"]) == O.ieee().max_rel_error(
        f, g["force_aos"])


def test_host_error_stats_match_numpy():
    from oracle import oracle as O
    g = golden("plummer4096")
    mx, rms = nb.force_error_stats(g["force_aos"], g["force_f64"][:, :3])
    mx2, rms2 = O.per_body_rel_error(g["force_aos"], g["force_f64"])
    assert abs(mx - mx2) <= 1e-12 and abs(rms - rms2) <= 1e-12


def test_newton3_refuses_more_bodies_than_it_evaluates():
    """Refused before anything is launched or read (the addresses are none)."""
    lib = _lib.load()
    limit = 65535 * 2048
    for n in (limit + 1, 1 << 28, 1 << 30):
        assert lib.nbgb_force_newton3_workspace_bytes(n) > 0
        assert lib.nbgb_force_newton3(1 << 20, 1 << 20, 1e-4, n, 1 << 20, 1 << 62, None) == -7, n
        assert lib.nbgb_force_newton3(1 << 20, 1 << 20, 1e-4, n, 1 << 20, 0, None) == -2, n


def test_kernels_launched_early_do_not_promise_read_only_data():
    """A kernel launched with programmatic dependence runs while the kernel
    before it still writes: no pointer to const among its parameters, or in
    the structs it takes, may be __restrict__ (loads through one may be
    non-coherent and may move ahead of the wait)."""
    src = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read())
           for p in glob.glob(os.path.join(ROOT, "nbody_gb300", "csrc", "*.cu*"))}
    everything = "\n".join(src.values())
    kernels = set()
    for m in re.finditer(r"launch_dependent(?:_n)?\(([^;]*?)\bst\b", everything):
        kernels |= set(re.findall(r"\b(\w+_kernel)\b", m.group(1)))
    assert len(kernels) >= 10, kernels
    read_only = re.compile(r"const\s+[\w:]+\s*\*\s*__restrict__")
    structs = set()
    for k in kernels:
        m = re.search(r"__global__[^;{]*?\b" + k + r"\s*\(([^{]*?)\)\s*\{", everything)
        assert m, k
        assert not read_only.search(m.group(1)), (k, m.group(1))
        structs |= set(re.findall(r"\b(\w*(?:Params|Integrate))\b", m.group(1)))
    structs |= {"Source"}  # held by the pair kernels' parameters
    assert {"Params", "ReduceParams", "DirectParams", "PairParams", "FusedIntegrate"} <= structs
    for name in structs:
        for text in src.values():
            if "launch_dependent" not in text and name != "FusedIntegrate":
                continue
            for m in re.finditer(r"struct " + name + r" \{(.*?)\n\};", text, flags=re.S):
                assert not read_only.search(m.group(1)), (name, m.group(1))
