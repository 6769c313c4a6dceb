"""Rules of the native sources whose breach no run shows reliably: read from the
source files (no GPU)."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "mojo-petsc4py_gb300" / "csrc"


def _code(name):
    """A source file without its comments."""
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", (CSRC / name).read_text(), flags=re.S)


def test_ring_writers_read_progress_by_acquire():
    """k_brick_sweep: a writer stores into slots of another tile's ring once that
    tile has published that it emptied them, so it reads the progress words
    (prog, rprog) by acquire, never by a plain or volatile load."""
    code = _code("gp_brick.cu")
    assert not re.search(r"volatile[^;{]*\bprog\b|volatile[^;{]*\brprog\b", code)
    body = code[code.index("__launch_bounds__(kBrickMaxThreads, 1) k_brick_sweep"):]
    body = body[:body.index("__global__")]
    for word, scope in (("prog", "progress"), ("rprog", "progress_cluster")):
        uses = re.findall(r"(\w*)\(?&" + word + r"\[", body)
        assert uses and set(uses) <= {scope, "publish", "cluster_map", "brick_relay", ""}
        assert scope in uses
    assert re.search(r"ld\.acquire\.cta\.shared\.b32", code)
    assert re.search(r"ld\.acquire\.cluster\.shared::cta\.b32", code)


def test_workspace_offsets_are_64_bit():
    """A solver's workspace is up to seven vectors of n < 2^31 doubles: an offset
    of several vectors is never a product of 32-bit integers."""
    for path in sorted(CSRC.glob("gp_*.cu")):
        code = _code(path.name)
        assert not re.findall(r"[+]\s*\(?[0-9]\s*\*\s*n\b", code), path.name
    code = _code("gp_ksp.cu")
    assert "return k->work + (size_t)i * k->n;" in code


def test_no_launch_status_is_dropped():
    """A captured pass keeps no kernel whose launch was refused: the status of each
    launch is looked at, in every source file."""
    for path in sorted(CSRC.glob("gp_*.cu*")):
        code = _code(path.name)
        assert not re.search(r"\(void\)\s*launch_pdl", code), path.name
        for call in re.finditer(r"(.{0,24})\blaunch_pdl\(", code, re.S):
            before = call.group(1).rstrip()
            assert before.endswith(("GP_CUDA(", "=", "cudaError_t")), (path.name, before)


def _before(code, start, end):
    code = code[code.index(start):]
    return code[:code.index(end)]


def test_captured_graphs_are_dropped_before_their_buffers():
    """A workspace or layout that a captured graph reads is rebuilt only after the
    graph is dropped and the mark of the old one cleared, so that an allocation that
    fails half-way leaves neither a graph of freed memory nor a half-built one taken
    for whole."""
    code = _code("gp_mixed.cu")
    for start, mark in (("static int mixed_buffers(", "M->n = M->m = 0;"),
                        ("static int mixed_factors(", "M->pc_generation = 0;"),
                        ("static int mixed_operator(", "M->adia_uid = 0;"),
                        ("static int mixed_blocks(", "M->bt_generation = 0;")):
        head = _before(code, start, "bt_build(" if "blocks" in start else "cudaFree(")
        assert "drop_pass(M);" in head and mark in head, start
    head = _before(_code("gp_ksp.cu"), "int ksp_solve(", "cudaGraphLaunch(")
    assert re.search(r"fit = ensure\(k, n, &moved\);\s*if \(moved \|\| fit != GP_OK\) drop_graph\(k\);",
                     head)
