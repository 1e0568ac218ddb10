"""The one-launch encoder deals a sentence's query rows to warps; a warp loads its first row before it looks at the others, so every item has
to begin inside the sentence.  The split is read out of the kernel's source and tried for every size that the kernel takes."""
import re
from pathlib import Path

SRC = (Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc" / "bert_small.cuh").read_text()


def test_items_begin_inside_the_sentence():
    stmt = re.search(r"const int (pairs = [^;]*);", SRC).group(1)
    parts = [p.split(" = ", 1) for p in re.split(r", (?=\w+ = )", stmt)]
    for t in range(1, 65):
        for ns in range(1, 64 // t + 1):
            env = {"a_t": t, "ns": ns, "CL": 16, "kBsThreads": 256, "kBsHeads": 12}
            for name, expr in parts:
                env[name] = eval(expr.replace("a.t", "a_t").replace("/", "//"), {"min": min, "max": max}, env)
            firsts = [k * env["per"] for k in range(env["split"])]
            assert all(f < t for f in firsts), (t, ns)
            assert firsts[-1] + env["per"] >= t
