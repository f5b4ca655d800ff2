"""Launch variants that the C-ABI takes by index: what include/lbrb.h says of
each index is what the dispatch launches for it."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_adjoint_variants_are_the_header_s():
    header = (ROOT / "include/lbrb.h").read_text()
    text = header[header.index("Launch variant of the two-step adjoint kernel"):header.index("int lbrb_adjoint_variants")]
    said = {int(i): (int(a), int(b), int(n)) for i, a, b, n in re.findall(r"(\d+): (\d+)x(\d+) (\d+)", text)}
    said |= {int(m[0]): tuple(map(int, m[1:])) for m in re.findall(r"(\d+): (\d+) (\d+) (\d+) (\d+)", text)}
    code = (ROOT / "lagrangianrbnudging_b200/csrc/adjoint_kernels.cu").read_text()
    code = code[code.index("switch (variant)"):]
    code = code[:code.index("}")]
    done = {}
    for case, args in re.findall(r"(case \d+|default): return launch_pair_t<Real, ([^>]*)>", code):
        tx, ty, threads, blocks = map(int, args.split(","))
        assert threads == tx * ty
        done[0 if case == "default" else int(case[5:])] = (tx, ty, blocks)
    for case, args, waves in re.findall(r"case (\d+): return launch_march_t<Real, ([^>]*)>\(P, (\d+), s\)", code):
        done[int(case)] = (*map(int, args.split(",")), int(waves))
    assert done == said
    assert sorted(done) == list(range(12))
    # the indices as they were given out: a caller's fixed variant keeps its launch
    assert [done[i] for i in range(4)] == [(32, 4, 4), (32, 4, 6), (32, 8, 2), (32, 8, 3)]
