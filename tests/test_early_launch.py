"""The surrogate's kernels that may start before the kernel ahead of them has ended
(launch_early) read what that one writes.  Only loads that griddepcontrol.wait orders
may do so: no read-only (non-coherent) ones, whose data must not change while the
kernel runs, and none that __restrict__ lets the compiler make read-only."""
import pathlib
import re

SRC = (pathlib.Path(__file__).resolve().parents[1] / "leven_gb300" / "csrc" / "lvn_surrogate.cu").read_text()
SRC = re.sub(r"//[^\n]*", "", SRC)


def function(name):
    """A function's text, from its return type to its closing brace."""
    m = re.search(rf"\b{name}\((?=[^;{{]*\)\s*{{)", SRC)
    start = SRC.rindex("\n__", 0, m.start())
    depth, i = 0, SRC.index("{", m.end())
    while True:
        depth += {"{": 1, "}": -1}.get(SRC[i], 0)
        i += 1
        if depth == 0:
            return SRC[start:i]


def test_early_kernels_read_nothing_as_constant():
    names = set(re.findall(r"launch_early\((k_\w+)", SRC))
    assert names == {"k_mlp_train", "k_adam_partials"}
    for name in sorted(names):
        text = function(name)
        assert "start_wait();" in text
        called = [c for c in set(re.findall(r"\b(\w+)\(", text)) if re.search(rf"__device__ [^;{{]*\b{c}\(", SRC)]
        for part in [text] + [function(c) for c in called]:
            assert not re.search(r"__ldg|__restrict__|ld\.global\.nc|ldca|__ldlu", part), (name, part[:120])
