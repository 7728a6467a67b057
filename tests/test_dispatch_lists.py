"""The micro-op kinds that the register kernels' jump tables list, taken from
the kernels' own sources: the switch of run_program (kernels_reg.cu) and of
run_forward/run_reverse (kernels_adj.cu) is compiled for the host with the
handlers replaced.  A kind outside its table is undefined behaviour on the
device, so every kind the encoder emits for an instance has to be listed."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

from rsr_b200 import evaluator as E
from test_dispatch_kinds import LEAF_MATVEC, STORE, UNARY, _programs

CSRC = Path(__file__).resolve().parents[1] / "rsr_b200" / "csrc"
F, FV3, FV2M2, FV3M3, ALL = range(5)
# the instances (profile, handler sets left out) that exist: reg_omittable, adj_omittable
REG = [(F, 0), (F, 1), (FV3, 0), (FV3, 1), (FV3, 2), (FV3, 3), (FV2M2, 0), (FV2M2, 1), (FV3M3, 0), (ALL, 0)]
ADJ = [i for i in REG if i[0] != ALL]

HOST = r"""
#include <stdio.h>
#include "uops.h"
using namespace rsr;
static int hit;
#define __builtin_unreachable() do { hit = 0; } while (0)
%s
template <int PROF, int OMIT> static void table(const char *name) {
    printf("%%s %%d %%d", name, PROF, OMIT);
    for (int k = 0; k < 256; ++k) {
        hit = 1;
        lists<PROF, OMIT>(k);
        if (hit) printf(" %%d", k);
    }
    printf("\n");
}
int main() { %s }
"""


def _defines(src, skip):
    """The RSR_ macros of a source, continuation lines included, but for `skip` (the handlers)."""
    out = re.findall(r"^#define RSR_(?:.*\\\n)*.*$", src, re.M)
    return "\n".join(d for d in out if not re.match(r"#define (?:%s)\(" % "|".join(skip), d))


def _reg(src):
    """run_program's switch: a case per kind, the stores and the stop included."""
    body = src[src.index("if constexpr (PROF == P_F && NU) {"):]
    body = body[:body.index("w = wn;")]
    return ("#define RSR_C(K) case (K): break;\n#define RSR_S(T) case kTapeKind[T]: break;\n" +
            _defines(src, ["RSR_C", "RSR_S"]) +
            "\ntemplate <int PROF, int OMIT> static void lists(int w) {\n"
            "    constexpr bool NU = (OMIT & 1) != 0, NM = (OMIT & 2) != 0; (void)NU; (void)NM;\n" + body + "}\n")


def _adj(src, extra):
    return ("#define KIND(K) case (K): break;\n" + _defines(src, ["RSR_F", "RSR_R"]) +
            "\ntemplate <class... T> static void tape_store(T...) {}\n"
            "template <int PROF, int OMIT> static void lists(int kind) { RSR_SWITCH(KIND, %s) }\n" % extra)


TAPES = "case kTapeKind[SF]: case kTapeKind[SV2]: case kTapeKind[SV3]: case kTapeKind[SM2]: case kTapeKind[SM3]: break;"


def _tables(tmp, text, instances):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    main = " ".join(f'table<{p}, {o}>("t");' for p, o in instances)
    (tmp / "t.cpp").write_text(HOST % (text, main))
    subprocess.run([cxx, "-std=c++17", "-O0", f"-I{CSRC}", "-o", str(tmp / "t"), str(tmp / "t.cpp")], check=True)
    rows = [r.split() for r in subprocess.run([str(tmp / "t")], check=True, capture_output=True,
                                              text=True).stdout.splitlines()]
    return {(int(r[1]), int(r[2])): {int(k) for k in r[3:]} for r in rows}


def _sources():
    reg, adj = (CSRC / "kernels_reg.cu").read_text(), (CSRC / "kernels_adj.cu").read_text()
    # the forward sweep's switch lists the tape stores that RSR_TAPES holds
    tapes = re.search(r"#define RSR_TAPES((?:.*\\\n)*.*)", adj).group(1)
    assert re.findall(r"case (kTapeKind\[\w+\]):", tapes) == [f"kTapeKind[{t}]" for t in ("SF", "SV2", "SV3", "SM2", "SM3")]
    return reg, adj


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    reg, adj = _sources()
    adj_lists = re.sub(r"#define RSR_TAPES(?:.*\\\n)*.*", "", adj)
    d = tmp_path_factory.mktemp
    return {"reg": _tables(d("reg"), _reg(reg), REG),
            "fwd": _tables(d("fwd"), f"#define RSR_TAPES {TAPES}\n" + _adj(adj_lists, "RSR_TAPES"), ADJ),
            "rev": _tables(d("rev"), _adj(adj_lists, "RSR_NONE"), ADJ)}


def _instance(prof, kinds):
    """The instance with the fewest handlers that a program of these kinds may run on (runtime.cu)."""
    omit = {F: 1, FV3: 3, FV2M2: 1}.get(prof, 0)
    if kinds & UNARY:
        omit &= ~1
    if kinds & LEAF_MATVEC:
        omit &= ~2
    return prof, omit


def _emitted():
    """(kernel, profile, kinds) of every program and form."""
    for p, nf in _programs():
        e = [int(w) for w in E.encoding(p, nf, 6)]
        if e[0] != 0xFFFFFFFF:
            yield "reg", e[0], {w & 255 for w in e[3:]}
        e = [int(w) for w in E.encoding(p, nf, 5)]
        if len(e) and e[0] <= FV3M3:
            n_fwd = e[7]
            yield "fwd", e[0], {w & 255 for w in e[9:9 + 2 * n_fwd:2]}
            yield "rev", e[0], {w & 255 for w in e[9 + 2 * n_fwd::2]}


def _missing(tables):
    out = set()
    for kernel, prof, kinds in _emitted():
        adj_kinds = kinds - STORE.keys() if kernel != "reg" else kinds
        prof, omit = _instance(prof, adj_kinds)
        for o in (omit, 0):
            out |= {(kernel, prof, o, k) for k in kinds - tables[kernel][prof, o]}
    return out


def test_every_emitted_kind_is_listed(tables):
    assert not _missing(tables)
    assert all(31 in t for kernel in tables.values() for t in kernel.values())   # the stop entry


def test_a_kind_taken_from_a_list_is_missed(tables, tmp_path):
    """The check itself: F+V3's list without its last kind, MAKE_VEC3."""
    src = _sources()[0].replace("RSR_C(K_V3 + 31) RSR_C(K_V3 + 33)", "RSR_C(K_V3 + 31)")
    short = dict(tables, reg=_tables(tmp_path, _reg(src), REG))
    assert {(k, p, kind) for k, p, _, kind in _missing(short)} == {("reg", FV3, 64 + 33)}
