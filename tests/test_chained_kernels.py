"""Kernels launched with launch_chained are resident while the kernel before
them still writes their inputs.  They must wait for it (chain_wait) and must not
read those inputs through the read-only path: ld.global.nc, __ldg, or a const
__restrict__ pointer, from which the compiler may derive either the same load or
the right to move it above the wait.  Read from the sources."""
import glob
import os
import re

import pytest

from conftest import ROOT

# tables that no kernel of a sweep writes: the triples' geometry, the folded
# expansion's operand
STATIC = {"tg", "xf"}
SOURCES = {f: open(f).read() for f in glob.glob(os.path.join(ROOT, "ddpcm_b200", "csrc", "*.cu"))}
CHAINED = sorted({k for s in SOURCES.values()
                  for call in re.findall(r"launch_chained\(([^;]*);", s)
                  for k in re.findall(r"\bk_\w+", call)})


def _close(text, i, pair="()"):
    """Index after the bracket that closes the one at text[i]."""
    depth = 0
    while True:
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        i += 1
        if depth == 0:
            return i


def _function(name):
    """(parameters, body) of the definition of `name`."""
    for s in SOURCES.values():
        for m in re.finditer(r"\b%s\(" % name, s):
            end = _close(s, m.end() - 1)
            if s[end:end + 2] == " {":
                return s[m.end():end - 1], s[end:_close(s, end + 1, "{}")]
    raise AssertionError(f"no definition of {name}")


def test_the_list_is_complete():
    assert CHAINED == ["k_extrap", "k_fold_proj", "k_fold_xi", "k_gram", "k_lx_gather", "k_lxs"]


@pytest.mark.parametrize("kernel", CHAINED + ["lxs_block"])
def test_inputs_of_a_sweep_take_ordinary_loads(kernel):
    params, body = _function(kernel)
    restricted = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert restricted <= STATIC, restricted - STATIC
    assert "__restrict__" not in body and ".nc" not in body and "__ldg" not in body
    if kernel != "lxs_block":
        assert "chain_wait();" in body


def test_read_only_loads_are_of_lists():
    lxs = next(s for f, s in SOURCES.items() if f.endswith("ddc_lxs.cu"))
    for m in re.finditer(r"ld\.global\.nc", lxs):  # in ld_list alone
        assert re.findall(r"__forceinline__ \w+ (\w+)\(", lxs[:m.start()])[-1] == "ld_list"
    assert re.findall(r"ld_list\(([\w.]+)", lxs.split("ld_list(const int* p)")[1]) == ["g.ls"]
