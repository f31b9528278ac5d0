"""A CTA of a cluster may touch another's shared memory only once that one is known to run: in every kernel that does, a wait at a
cluster barrier comes before the first such access.  Read from the source, because a kernel without it mostly works."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mdi_llm_b200" / "ops" / "csrc"
REMOTE = re.compile(r"\b(?:mapa|st_cluster\w*|cluster_addr|mbar_arrive_cta|tcgen05_commit_pair)\b")
WAIT = re.compile(r"barrier\.cluster\.wait|\bcluster_sync_all\s*\(")


def _kernels(text):
    """(name, body) of the __global__ functions of a source file, without comments."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"__global__", text):
        at = text.index("{", m.start())
        name = re.findall(r"(\w+)\s*\(", text[m.start():at].replace("__launch_bounds__", "").replace("__cluster_dims__", ""))[-1]
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield name, text[at:end]


FOUND = [(f.name, name, body) for f in sorted(CSRC.glob("*.cu")) for name, body in _kernels(f.read_text()) if REMOTE.search(body)]


def test_the_kernels_are_found():
    assert {"few_rows_linear_kernel", "attn_decode_kernel", "gemm_fp8_kernel", "gemm_bf16_tcgen05_kernel",
            "gemm_bf16_tcgen05_pair_kernel"} <= {name for _, name, _ in FOUND}


@pytest.mark.parametrize("source,name,body", FOUND, ids=[f"{n}" for _, n, _ in FOUND])
def test_a_cluster_is_waited_for_before_it_is_written_to(source, name, body):
    wait = WAIT.search(body)
    assert wait and wait.start() < REMOTE.search(body).start()
