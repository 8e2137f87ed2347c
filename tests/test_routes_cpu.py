"""Rules that choose between forms of a kernel, compiled from their source and asked about sizes at which both forms were timed."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "mesh_llm_b200", "csrc")

PRELUDE = """
#include <cstdint>
#include <cstdio>
#include <cstdlib>
static int64_t kq_div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }
static int kq_sm_count() { return 148; }
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    """(rule, a, b) -> its answer for two numbers"""
    with open(os.path.join(CSRC, "kq_stage.cu")) as f:
        s = f.read()
    consts = "".join(re.search(r"^constexpr int " + n + r" = [^;]*;", s, re.M).group(0) + "\n" for n in ("ROUTER_TILE", "RB"))
    rules = ["router_takes_blocks", "router_fused_rows"]
    code = PRELUDE + consts + "".join(re.search(r"^\w+ " + n + r"\(.*?}\n(?=\S)", s, re.M | re.S).group(0) for n in rules)
    code += "int main(int, char **v) {\n" + "".join(f'    if (v[1][0] == \'{i}\') printf("%d", (int){n}(atoll(v[2]), atoll(v[3])));\n' for i, n in enumerate(rules)) + "}\n"
    d = tmp_path_factory.mktemp("routes")
    (d / "r.cpp").write_text(code)
    subprocess.run(["g++", "-std=c++17", str(d / "r.cpp"), "-o", str(d / "r")], check=True)
    return lambda rule, a, b: int(subprocess.run([str(d / "r"), str(rules.index(rule)), str(a), str(b)], check=True, capture_output=True, text=True).stdout)


@pytest.mark.parametrize("T,E,blocks", [(1024, 128, 1), (2048, 64, 1), (2048, 128, 1), (4096, 32, 1), (4096, 96, 1), (4096, 160, 1), (2048, 8, 0), (2048, 16, 0), (2048, 32, 0), (2048, 33, 0),
                                        (1024, 33, 0), (512, 128, 0), (512, 160, 0), (1024, 160, 0), (2048, 65, 0), (2048, 160, 0), (4096, 8, 0), (4096, 33, 0), (4096, 65, 0), (9, 8, 0)])
def test_router_logits_by_blocks(ask, T, E, blocks):
    """blocks of 32 tokens x 32 experts only where they were the faster form"""
    assert ask("router_takes_blocks", T, E) == blocks


@pytest.mark.parametrize("E,h,rows", [(128, 2048, 24), (8, 2048, 24), (128, 4096, 24), (64, 4096, 24), (32, 1024, 24), (256, 2048, 16), (256, 7168, 16), (256, 8192, 16), (160, 6144, 16), (16, 512, 8)])
def test_rows_of_the_one_launch_routing(ask, E, h, rows):
    """as many rows as the one launch was the faster form for; 8 and fewer have a rule of their own"""
    assert ask("router_fused_rows", E, h) == rows
