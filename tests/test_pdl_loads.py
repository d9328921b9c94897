"""Kernels that are launched before their predecessors have finished must not
claim that their inputs are read-only (csrc/pdl.cuh).

A kernel that calls pdl_enter() is resident while earlier kernels of the stream
write what it will read. __ldg, ld.global.nc and __restrict__ promise memory
that nothing writes during the kernel: only the resident twiddle tables
(uint2) are. This reads the sources; no GPU is needed."""
import os
import re

import pytest

import b200mul

CSRC = os.path.join(os.path.dirname(b200mul.LIB_PATH), "csrc")
# the transforms of the 64-bit field: ordinary launches
ORDINARY = {f for f in os.listdir(CSRC) if f.startswith("ntt_")} | {"b2m_field.cu"}
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")) and f not in ORDINARY)


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _closing(text, start, pair):
    """Index after the bracket that closes the one at `start`."""
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def _functions(text):
    """(name, parameters, start and end of the body) of every function."""
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        if m.group(1) in ("if", "for", "while", "switch", "return", "sizeof", "asm"):
            continue
        try:
            end = _closing(text, m.end() - 1, "()")
        except ValueError:
            continue
        brace = re.match(r"\s*(?:const\s*)?\{", text[end:])
        if brace:
            body = end + brace.end() - 1
            yield m.group(1), text[m.end():end - 1], body, _closing(text, body, "{}")


def _launched_early():
    """Kernels given to launch_pdl."""
    names = set()
    for f in FILES:
        text = _source(f)
        for m in re.finditer(r"\blaunch_pdl\(", text):
            names |= set(re.findall(r"\bk_\w+", text[m.end():_closing(text, m.end() - 1, "()")]))
    return names


def test_kernels_launched_early_wait_first():
    early, bodies = _launched_early(), {}
    for f in FILES:
        text = _source(f)
        bodies.update({fn: text[i:j] for fn, _, i, j in _functions(text)})
    waits = {fn for fn, body in bodies.items() if "pdl_enter();" in body}
    assert {"k_rns_carry", "k_rns_first", "k_rns_small", "k_school", "k_shl", "k_dc_fix", "k_residues"} <= early
    for k in early:
        assert k in waits or re.search(r"\b(%s)\b" % "|".join(waits), bodies[k]), k
    assert not any("pdl" in _source(f) for f in ORDINARY)


@pytest.mark.parametrize("name", FILES)
def test_only_tables_are_read_as_read_only(name):
    text = _source(name)
    functions = list(_functions(text))
    for m in re.finditer(r"__ldg|ld\.global\.nc", text):
        owner = {fn for fn, _, i, j in functions if i <= m.start() < j}
        assert owner and owner <= {"rns_ld", "rns_ld2", "rns_ld4"}, owner
    early = _launched_early()
    for fn, params, i, j in functions:
        if fn not in early and re.search(r"__global__[^;{}]*\b%s\s*\(" % fn, text):
            continue  # an ordinary launch starts after its predecessors' ends
        for p in params.split(","):
            assert "__restrict__" not in p or "uint2" in p, (fn, p.strip())
