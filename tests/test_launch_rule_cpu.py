"""Kernels that begin beside the launch before them (launch_wait in csrc/pw_common.cuh) reach its data, and write their
outputs, through pointers without __restrict__: the qualifier would let a compiler move an access across the wait.  Read
off the sources: a kernel with a wait, or a device function that one hands its planes to, keeps __restrict__ only on the
inputs listed here, each complete before the predecessor begins."""

import glob
import os
import re

import pytest

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")

# tables, V(r) and maps of the handle; blocks written two launches earlier or more
COMPLETE = {
    "k_plane": {"vz", "twx", "twy"}, "k_plane_rt": {"vz", "twx", "twy"},
    "k_zi": {"col_start", "col_lo", "tw"}, "k_zf": {"psi", "kin", "col_start", "col_lo", "tw"},
    "k_pack_pairs": {"half_idx", "half_neg"}, "k_resid_column": {"kin"},
    "k_block_nl": {"B", "psi", "ch_atom", "atom_ch_start", "d_off", "d_vals"}, "k_block_p": {"Pn", "HPn"},
    "k_block_update": {"B", "HB", "cols", "pcols"}, "k_eigh_cluster": set(),
    "plane_ya": set(), "plane_yd": set(),
}


def _functions():
    """(name, parameter list, body) of every kernel and plane pass in the sources."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"\b(k_\w+|plane_y\w)\s*\(((?:[^(){};]|\([^()]*\))*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield m.group(1), m.group(2), text[m.end():i]


def test_every_waiting_kernel_is_listed():
    waiting = {n for n, _, body in _functions() if "launch_wait()" in body}
    assert waiting == {n for n in COMPLETE if n.startswith("k_")}


@pytest.mark.parametrize("name", sorted(COMPLETE))
def test_only_complete_inputs_are_restrict(name):
    found = [p for n, p, _ in _functions() if n == name]
    assert found
    for params in found:
        restrict = set(re.findall(r"__restrict__\s+(\w+)", params))
        assert restrict <= COMPLETE[name]
        outputs = {re.search(r"(\w+)\s*$", p).group(1) for p in params.split(",") if "*" in p and "const" not in p}
        assert not outputs & restrict
