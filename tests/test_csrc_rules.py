"""Rules that the kernels' sources keep and that no run can show to be broken without harm: read from the text, on the CPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "v620-inference-engine_b200", "ops", "csrc")


def _text(path):
    """Source without comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def _kernels(path):
    """(name, body) of every kernel of a file; a body ends where its braces do."""
    t = _text(path)
    for m in re.finditer(r"__global__[^;{]*?(\w+)\(", t):
        at = depth = t.index("{", t.index(")", m.end()))
        end, depth = at, 0
        while True:
            depth += {"{": 1, "}": -1}.get(t[end], 0)
            end += 1
            if depth == 0:
                break
        yield m.group(1), t[at:end]


def _sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def test_a_cluster_meets_before_one_block_reaches_into_another():
    """Shared memory of another block of the cluster may be used only when that block has begun to run."""
    seen = 0
    for path in _sources():
        for name, body in _kernels(path):
            first = body.find("map_shared_rank")
            if first < 0:
                continue
            seen += 1
            handle = re.search(r"(\w+)\s*=\s*cg::this_cluster\(\)|cg::cluster_group (\w+)", body)
            sync = body.find(next(g for g in handle.groups() if g) + ".sync()")
            assert 0 <= sync < first, (os.path.basename(path), name)
    assert seen >= 3


def test_waits_before_warp_wide_instructions_are_voted_on():
    """Lanes come out of a polling loop one by one and may even disagree on its outcome; every wait is one verdict for the warp, and
    tensor memory is read only after the warp has come together."""
    for path in _sources():
        t = _text(path)
        calls = re.findall(r"\b(?:mbar_wait|mg_wait)\((?!uint64_t)", t)
        inside = re.findall(r"__all_sync\(0xffffffffu, (?:mbar_wait|mg_wait)\(", t)
        assert len(calls) == len(inside), os.path.basename(path)
        for fn in re.findall(r"__device__ __forceinline__ void tmem_ld\w+\(uint32_t taddr[^{]*\{([^}]*)", t):
            assert fn.lstrip().startswith(("__syncwarp();", "tmem_ld")), os.path.basename(path)
    # no lane skips to the next warp-wide load by itself: a lane's row or column only guards its stores
    for name in ("moe_tc.cu", "vit_attn.cu", "gemm_tc.cu"):
        t = _text(os.path.join(CSRC, name))
        for m in re.finditer(r"tcgen05\.wait::ld\.sync\.aligned[^\n]*\n([^\n]*)", t):
            assert not re.search(r"if \((?:row|col)\b.*\) continue;", m.group(1)), (name, m.group(1))


@pytest.mark.parametrize("name", sorted(os.path.basename(p) for p in _sources()))
def test_divisions_are_rounded_like_any_other_operation(name):
    """Sigmoids and the like that were formed with a correctly rounded division stay so."""
    assert "__fdividef" not in _text(os.path.join(CSRC, name))
