"""The overflow flags while a plan on another stream may set them: a kernel of the
batch DAG that runs beside such a plan and whose threads meet at a barrier, a vote or
a shuffle reads them once for the CTA (any_overflow), so that no thread returns alone.

The kernels that run beside a plan of another stream are those of the DAG's table
stream and of its main stream up to the join with the quads (enqueue_fresh_dag and
enqueue_mesh_dag in lvn_api.cu); the quad stream's own kernels follow both plans."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "leven_gb300" / "csrc"
SRC = re.sub(r"//[^\n]*", "", (CSRC / "lvn_kernels.cu").read_text())
API = (CSRC / "lvn_api.cu").read_text()
MEET = re.compile(r"__syncthreads|__syncwarp|_sync\(")


def body(text, at):
    depth, i = 0, text.index("{", at)
    start = i
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def functions():
    out = {}
    for m in re.finditer(r"__(?:device|global)__[^;{}]*?\b(\w+)\((?:[^(){};]|\([^(){};]*\))*\)\s*(?:const\s*)?\{", SRC):
        out.setdefault(m.group(1), "")
        out[m.group(1)] += body(SRC, m.end() - 1)
    return out


def launched(launcher):
    """The kernels a launch_* function launches."""
    return set(re.findall(r"\b(k_\w+)\s*(?:<[^<>;]*>)?\s*<<<", body(SRC, SRC.index(f"cudaError_t {launcher}("))))


def test_flags_read_once_beside_a_plan():
    fresh, mesh = (body(API, API.index(f"int {n}(lvn_meshgen* m")) for n in ("enqueue_fresh_dag", "enqueue_mesh_dag"))
    main = set(re.findall(r"(launch_\w+)\(\w+, s0\)", fresh[fresh.index("ev_plan"):]))
    main |= set(re.findall(r"(launch_\w+)\(\w+, s0\)", mesh[:mesh.index("cudaStreamWaitEvent(s0, m->ev_mesh")]))
    tables = set(re.findall(r"(launch_\w+)\(\w+, tab\)", mesh))
    assert main == {"launch_edge_scatter", "launch_hermite", "launch_leaf"}
    assert tables == {"launch_primes", "launch_hash_fill", "launch_edge_insert", "launch_node_insert"}
    fns = functions()

    def meets(name, seen):
        if name in seen or name not in fns or name == "any_overflow":
            return False
        seen.add(name)
        return bool(MEET.search(fns[name])) or any(meets(c, seen) for c in set(re.findall(r"\b(\w+)\s*(?:<[^<>;()]*>)?\(", fns[name])))

    kernels = set().union(*(launched(n) for n in main | tables))
    assert {"k_hermite", "k_hermite_smem", "k_hermite_wide", "k_leaf", "k_primes", "k_hash_repair"} <= kernels
    for k in sorted(kernels):
        if "overflow" not in fns[k] or not meets(k, set()):
            continue
        assert "if (any_overflow(b)) return;" in fns[k], k
        assert "bs->overflow" not in fns[k], k
