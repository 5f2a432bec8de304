"""Kernels launched as dependents (csrc/common.cuh, launch_dep) start while the
kernel directly before them still writes.  What that kernel writes must not be
read through the read-only path, which promises data that is constant from the
kernel's first instruction and which the compiler may read ahead of the wait.
Read from the sources: every read-only access of a kernel that calls grid_wait
names data that is older than its predecessor, or constant.  CPU only."""

import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "dpmd-public_gb300", "csrc")

# const __restrict__ parameters: plan and frame tables, statistics, index
# arrays of the batch, and what was written before the direct predecessor
# began (the env build's earlier kernels; everything before the clear that
# k_localize, k_scatter_atomic and k_virial_pairs follow)
READ_ONLY = {
    "k_localize": {"fr", "coord", "atype"},
    "k_cell_scan": {"fr"},
    "k_cell_bucket": {"fr", "atom_frame", "atom_cell"},
    "k_cell_rank": {"fr", "atom_frame", "atom_cell", "cell_start", "cell_count", "atom_sub"},
    "k_ghost_fill": {"fr", "cell_start", "cell_count", "ext_start", "ghost_start"},
    "k_nlist_env": {"fr", "atom_frame", "atom_cell", "atom_sub", "ext_sub", "atype", "avg", "stdv"},
    "k_nlist_env_ext": {"avg", "stdv"},
    "k_emb_dx16": {"drow"},
    "k_frame_energy_cta": {"frame_of_row"},
    "k_scatter_atomic": {"net", "dR", "rij", "nlist"},
    "k_virial_pairs": {"net", "dR", "rij", "nlist"},
}
# first name of every __ldg argument in a file with dependent launches: weights
# and parameters (src, cs), F1's row scales (F1 follows a clear), the inputs of
# the two prod kernels (p: V4::load4), rows of 1 / dstd
LDG = {
    "embed_tc.cu": {"src"},
    "fit_tc.cu": {"src", "cs", "ep"},
    "prod.cu": {"p", "nlist", "rij"},
    "desc_blk.cu": set(),
    "env.cu": set(),
}
# helpers on ld.global.nc and what the dependent kernels may give them
NC = {"desc_blk.cu": {"ld_tab4": {"row", "r"}, "ld_row4": {"isd"}}}


def _kernels(src):
    for m in re.finditer(r"__global__", src):
        j = src.index("{", m.start())
        depth, k = 0, j
        while True:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            if depth == 0:
                break
            k += 1
        head = src[m.start():j]
        yield re.search(r"\b(k_\w+)\s*\(", head).group(1), head, src[j:k + 1]


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def test_dependent_kernels_read_older_data_read_only():
    seen = set()
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for name, head, body in _kernels(_code(path)):
            if "grid_wait()" not in body:
                continue
            seen.add(name)
            got = set(re.findall(r"const [^,()]*?\*\s*__restrict__ (\w+)", head))
            assert got <= READ_ONLY.get(name, set()), (name, got)
    assert {"k_fwd_blk", "k_bwd_blk", "k_emb_fwd", "k_nlist_env", "k_fx_finish2"} <= seen


def test_read_only_loads_name_constants():
    for f, allowed in LDG.items():
        src = _code(os.path.join(CSRC, f))
        got = set(re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?(\w+)", src))
        assert got <= allowed, (f, got)
    nc = r"\b(ld_(?:tab|stream|first|row)\d?)\(\s*(\w+)"
    for f, allowed in NC.items():
        src = _code(os.path.join(CSRC, f))
        src = re.sub(r"__device__[^{]*", "", src)  # (the helpers' own definitions)
        for fn, arg in re.findall(nc, src):
            assert arg in allowed.get(fn, set()), (f, fn, arg)


def test_loads_of_the_previous_kernels_data_stay_after_the_wait():
    src = _code(os.path.join(CSRC, "fused.cuh"))
    got = re.findall(r"(float4?) ld_prev4?\(const float\* p\) \{(.*?)\n\}", src, flags=re.S)
    assert len(got) == 2
    for _, body in got:
        assert "asm volatile(\"ld.global.L1" in body and ": \"memory\")" in body
