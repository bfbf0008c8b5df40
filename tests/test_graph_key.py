"""The batch graph is captured again when anything its kernels and copies were given
has changed: its key holds every buffer of the kernels' arguments (BatchPtrs), or the
arguments as a whole, and the host buffers of its copies."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "leven_gb300" / "csrc"


def test_key_holds_every_buffer():
    api = (CSRC / "lvn_api.cu").read_text()
    make = api[api.index("BatchPtrs make_ptrs("):]
    make = make[:make.index("\n}\n")]
    pools = set(re.findall(r"b\.(\w+) = m->\w+\.as<", make))
    assert {"desc", "planes", "hmap", "search", "quad_scratch", "leaf_qef"} <= pools and len(pools) > 25
    key = api[api.index("std::vector<uintptr_t> key"):api.index("key != m->graph_key")]
    whole = "std::memcpy(key.data(), &b, sizeof(b));" in key and "std::memset(&b, 0, sizeof(b));" in make
    members = dict(re.findall(r"b\.(\w+) = m->(\w+)\.as<", make))
    missing = [p for p in sorted(pools) if not whole and f"m->{members[p]}.p" not in key and f"(uintptr_t)b.{p}," not in key]
    assert not missing, missing
    copies = api[api.index("int enqueue_inputs("):api.index("int upload(")] + \
        api[api.index("int enqueue_state_readback("):api.index("int finish_states(")]
    for host in set(re.findall(r"m->(h_\w+)\.p", copies)):
        assert f"m->{host}.p" in key, host
