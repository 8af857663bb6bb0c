"""Kernels that are launched early (griddepcontrol: the launch before may still be
writing) read what that launch writes by coherent loads behind the wait, never
through the non-coherent path, whose loads need data that is constant for the
kernel's lifetime and may be moved above the wait.

Which launch writes what follows from the chains (plane_fwd, pencil, plane_inv):
a plane_fwd reads its field and its prologue's arrays right after any writer, a
pencil pass reads the scalars of the plane_fwd before it; what an epilogue reads
beside its transform is at least two launches old. So __ldg may appear in the
tables (twiddles, symbols) and in the epilogues, and nowhere else. Read from the
sources: such a load gives the right value on almost every run."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "spm-iqc_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _structs(code):
    """(name, body) of every top-level policy struct of ops.cuh."""
    out = []
    for m in re.finditer(r"\bstruct (\w+) \{", code):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
        out.append((m.group(1), code[m.end():i]))
    return out


def test_no_noncoherent_loads_outside_the_tables():
    for name in ("fft_core.cuh", "fft_kernels.cuh", "tile_kernels.cuh"):
        code = _code(name)
        assert ".nc" not in code, name
        for line in code.splitlines():
            if "__ldg(" in line:
                assert re.search(r"__ldg\((symtab_of|gtab_of)\(", line), (name, line)


def test_prologues_and_operators_use_coherent_loads():
    code = _code("ops.cuh")
    seen = set()
    for name, body in _structs(code):
        kind = re.match(r"Pro|Op|Epi", name)
        if kind and kind.group() != "Epi":
            seen.add(kind.group())
            assert "__ldg(" not in body and "scal_in(" not in body, name
    assert seen == {"Pro", "Op"}
    # nothing else in the file hides such a load
    rest = code
    for _, body in _structs(code):
        rest = rest.replace(body, "")
    assert rest.count("__ldg(") == 1 and "scal_in" in rest  # scal_in itself


def test_scalars_of_the_launch_before_are_read_behind_the_wait():
    """Operators that need such a scalar name it (PRE), and the pencil pass reads it
    after grid_dep_sync with a volatile load."""
    code = _code("ops.cuh")
    pre = {n for n, b in _structs(code) if re.search(r"\bPRE\b", b)}
    assert pre == {"OpForce", "OpTangent"}
    tile = _code("tile_kernels.cuh")
    pencil = tile[tile.index("pencil_kernel("):]
    wait, load = pencil.index("grid_dep_sync()"), pencil.index("PreOf<Op>::value >= 0")
    assert wait < load and "volatile const double" in pencil[load:load + 120]


def test_flow_words_are_read_behind_the_wait():
    body = _code("fft_core.cuh").split("bool flow_state(")[1].split("\n}")[0]
    assert "__ldcg" not in body and "volatile" in body
