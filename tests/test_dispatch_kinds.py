"""The register kernels dispatch through a jump table without a range check
(kernels_reg.cu run_program, kernels_adj.cu run_forward/run_reverse): every
micro-op kind the encoder emits for a profile must be one its table lists."""
import pytest

from programs import kat_cases, single_op_programs
from rsr_b200 import evaluator as E
from rsr_b200 import isa as I
from rsr_b200 import workloads as W
from rsr_b200.generator import Generator, OpSet

F = set(range(27))
V2, V3, M2, M3 = (set(range(b, b + n)) for b, n in ((32, 27), (64, 34), (104, 27), (136, 27)))
UNARY = set(range(21, 27))
LEAF_MATVEC = {64 + 30, 64 + 31, 64 + 32}   # matrix from a feature, a constant, a stack slot
# accumulator types of each profile (uops.h kProfileTypes) and the kinds of its full table;
# F+V3 has no Mat3 accumulator to multiply from or to spill
TABLE = {0: F, 1: F | V3 - {64 + 29, 64 + 32}, 2: F | V2 | M2, 3: F | V3 | M3, 4: F | V2 | V3 | M2 | M3}
OMITTABLE = {0: [UNARY], 1: [UNARY, LEAF_MATVEC], 2: [UNARY], 3: [], 4: []}
TAPE = {0: {27}, 1: {27, 98}, 2: {27, 59, 131}, 3: {27, 98, 163}}

STORE = {27: 1, 59: 2, 98: 3, 131: 4, 163: 9}   # a prologue's stores: components of the type


def _reads_feature(w):
    """Whether a word of the accumulator form has a feature operand (uops.h)."""
    t = max(b for b in (0, 32, 64, 104, 136) if b <= w & 255)
    k, arg = (w & 255) - t, w >> 8
    nb = {0: 6, 32: 3}.get(t, 5)
    if (w & 255) in STORE or k == 1:
        return False
    if k == 0:
        return True
    if k == 2:                                # a load after a PUSH
        return (arg >> 4) & 7 != 0 and (arg >> 7) & 1 == 0
    if k < 3 + 3 * nb:
        return (k - 3) % 3 == 0
    k -= 3 + 3 * nb
    if t == 0:                                # unary: bits 12-13 load first
        return (arg >> 12) & 3 == 1
    if k < 4:
        return k == 1                         # SCALE {A X C S}
    if t in (32, 64):
        w3 = t == 64
        if k < 7:
            return k == 4                     # DOT {X C S}
        if k < 10 + w3:
            return (arg >> 12) & 3 == 1       # NORM, GET
        return k == 11 + w3                   # MULM {A X C S}, MAKE
    return k < 8 and (arg >> 12) & 3 == 1     # DET TRACE TRANSPOSE INVERSE, MAKE


def _mixed(types, n, seed):
    """Random programs over every operator whose operands and result are of `types`."""
    ops = [o for o in I.BASIC_NAMES + I.LINALG_NAMES if {*I.SIGNATURE[o][0], I.SIGNATURE[o][1]} <= set(types)]
    off = {I.FLOAT: 0, I.VEC2: 1, I.VEC3: 3, I.MAT2: 6, I.MAT3: 10}
    gen = Generator(OpSet(ops, [(t, off[t]) for t in types], list(types), 1.0), seed)
    return [(p, 19) for p in gen.population(n, 1, 60)]


def _programs():
    out = [(p, ds.num_features) for p, ds, _ in kat_cases(16).values()]
    out += [(p, 19) for p in single_op_programs().values()]
    for pop, nf in ((W.scalar_population(200), 1), (W.lorentz_population(300), 9), (W.transform_population(200), 15),
                    (W.inverse_population(200), 8)):
        out += [(p, nf) for p in pop]
    for types, seed in (((I.FLOAT,), 1), ((I.FLOAT, I.VEC3), 2), ((I.FLOAT, I.VEC2, I.MAT2), 3),
                        ((I.FLOAT, I.VEC3, I.MAT3), 4), ((I.FLOAT, I.VEC2, I.VEC3, I.MAT2, I.MAT3), 5)):
        out += _mixed(types, 300, seed)
    return out


@pytest.mark.parametrize("form", [1, 5, 6])
def test_every_emitted_kind_is_in_its_profiles_table(form):
    seen = {}
    for p, nf in _programs():
        if form == 1:
            prof = E.analyze(p, nf)["fast_profile"]
            if prof < 0:
                continue
            kinds = {int(w) & 255 for w in E.encoding(p, nf, 1)}
            table = TABLE[prof]
        elif form == 6:   # constant subtrees hoisted: prologue, stop, main program
            e = [int(w) for w in E.encoding(p, nf, 6)]
            prof, main, n_hoist, code = e[0], e[1], e[2], e[3:]
            if prof == 0xFFFFFFFF:
                continue
            table = TABLE[prof]
            stores = [w for w in code[:main] if (w & 255) in STORE]
            assert sorted(i for w in stores for i in range(w >> 8, (w >> 8) + STORE[w & 255])) == \
                list(range(p.param_count(), p.param_count() + n_hoist))
            assert (main == 0) == (n_hoist == 0) and (main == 0 or code[main - 1] == 31)
            # nothing in a prologue depends on the point
            assert not any(_reads_feature(w) for w in code[:max(main - 1, 0)])
            kinds = {w & 255 for i, w in enumerate(code) if i != main - 1} - STORE.keys()
        else:
            e = E.encoding(p, nf, 5)
            prof = int(e[0]) if len(e) else 4
            if prof not in TAPE:   # not the register adjoint's
                continue
            code = e[7:]
            n_fwd, n_rev = int(code[0]), int(code[1])
            assert len(code) == 2 + 2 * (n_fwd + n_rev)   # where the kernel puts its stop entries
            kinds = {int(w) & 255 for w in code[2::2]}
            table = TABLE[prof] | TAPE[prof]
        assert kinds <= table, (prof, sorted(kinds - table))
        # leaving out a handler set whose kinds do not occur keeps every kind that does
        for gone in OMITTABLE[prof]:
            assert kinds & gone or kinds <= table - gone
        seen[prof] = seen.get(prof, 0) + 1
    assert set(seen) == (set(TAPE) if form == 5 else set(TABLE)) and min(seen.values()) >= 50, seen
