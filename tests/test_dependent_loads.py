"""Kernels that are launched as programmatic dependents may be resident before the kernel before them
has ended, so that what that one writes is not read-only while they run: their code has no load of
the read-only path (ld.global.nc, __ldg)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "helio_b200" / "csrc"


def code(name: str) -> str:
    text = (CSRC / name).read_text()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_dependent_launches_read_nothing_through_the_read_only_path():
    dependents = [p.name for p in CSRC.glob("*.cu") if re.search(r"launch_after\(|ProgrammaticStreamSerialization", code(p.name))]
    assert {"hiz.cu", "instance_cull.cu", "shadow_cull.cu", "vg_build.cu", "vg_cull.cu", "batch.cu"} == set(dependents)
    texts = {n: code(n) for n in dependents if n != "batch.cu"}
    texts.update({p.name: code(p.name) for p in CSRC.glob("*.cuh")})
    # Of the batch only the packing is a dependent launch; its two cooperative kernels are not.
    batch = code("batch.cu")
    assert batch.count("launch_after(") == 1
    start = batch.index("pack_draws_kernel(")
    texts["batch.cu"] = batch[start:batch.index("cudaError_t launch_pack_draws(")]
    for name, text in texts.items():
        assert not re.search(r"__ldg\(|\.nc\b", text), name
        for head, body in re.findall(r"__global__([^;{]*)\{(.*?)\n\}", text, flags=re.S):
            assert "pdl_wait()" in body or "instance_cull_data_kernel" in head, (name, head)
