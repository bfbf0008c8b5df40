"""Tensor-memory columns of the training kernel's last contractions: a gradient that
is written out while the next product runs is read from columns that product does not
write.  The products, reads and column numbers are taken from the source."""
import pathlib
import re

SRC = (pathlib.Path(__file__).resolve().parents[1] / "leven_gb300" / "csrc" / "lvn_surrogate.cu").read_text()
HIDDEN, IN, ONES = 128, 96, 16


def column(name):
    return int(re.search(rf"constexpr uint32_t {name} = (\d+);", SRC).group(1))


def width(name):
    """Columns a tensor-memory load takes."""
    body = SRC[SRC.index(f" {name}("):]
    return int(re.search(r"32x32b\.x(\d+)", body).group(1))


def test_reads_beside_products():
    assert re.search(r"kIdescDW = umma_idesc\(kHidden, kHidden \+ 16\)", SRC)
    assert re.search(r"kIdescDW0 = umma_idesc\(kHidden, kIn \+ 16\)", SRC)
    flush = SRC[SRC.index("auto flush = [&]"):]
    flush = flush[:flush.index("\n    };")]
    weights, bias = flush.split("if (cq == 0)")
    load = re.compile(r"(tmem_ld32|tmem_issue16)\(tmem \+ col0 \+ (tl|in)")
    assert load.findall(weights) == [("tmem_ld32", "tl")] and width("tmem_ld32") == 32
    (name, at), = load.findall(bias)
    assert at == "in"
    products = {"dW1": range(column("kTmDW1"), column("kTmDW1") + HIDDEN + ONES),
                "dW0": range(column("kTmDW0"), column("kTmDW0") + IN + ONES)}
    for tiles in (1, 2, 3, 5):
        reads = {0: ["kTmDW2"], 1: ["kTmDW3"]}  # by the product they run beside (the loop over the items)
        reads.setdefault(tiles, []).append("kTmDW1")
        for item, gradients in reads.items():
            product = products["dW1" if item < tiles else "dW0"]
            for g in gradients:
                first = column(g)
                read = set(range(first, first + HIDDEN)) | set(range(first + HIDDEN, first + HIDDEN + width(name)))
                assert not read & set(product), (tiles, item, g)
                assert max(read) < 512
