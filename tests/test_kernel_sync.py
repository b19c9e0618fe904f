"""Orderings that a run cannot be relied on to miss (CPU, from the kernels'
source): what one thread writes to shared memory another may read only past a
barrier that both take part in."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paising_gb300", "csrc")


def kernel_body(file: str, name: str) -> str:
    """The body of kernel `name`, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    at = re.search(r"__global__[^;{]*\b" + name + r"\(", text)
    assert at, f"{name} not in {file}"
    start = text.index("{", at.end())
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError(f"{name}: unbalanced braces")


@pytest.mark.parametrize("file,name,access", [
    ("pa_resample.cu", "resample_fused_kernel", r"remote\(\w+, r\)\["),
    ("pa_msc_cluster.cu", "msc_sweep_cluster_kernel", r"map_shared_rank\(")])
def test_cluster_starts_before_its_shared_memory_is_used(file, name, access):
    """Another CTA's shared memory exists once that CTA has started, which only
    a barrier of the whole cluster shows: one is completed (sync, or arrive and
    then wait) before the first access."""
    body = kernel_body(file, name)
    first = re.search(access, body)
    assert first
    before = body[:first.start()]
    before = re.sub(r"auto cluster_sync = .*?};", "", before, flags=re.S)  # a definition, not a barrier
    arrive, wait = before.find("barrier_arrive()"), before.rfind("barrier_wait()")
    assert "cluster.sync()" in before or "cluster_sync()" in before or 0 <= arrive < wait


def test_adaptive_step_hands_its_temperature_on_in_order():
    """The thresholds of a new temperature are formed by twelve lanes from the
    value one lane chose.  Shuffles order no memory: past the block's last
    barrier no shared memory is written by one lane for the others."""
    body = kernel_body("pa_resample.cu", "adapt_kernel")
    shared = set()
    for decl in re.findall(r"__shared__\s+(?:double|bool|int|uint32_t)\s+([^;]*);", body):
        shared |= {re.match(r"\w+", v.strip()).group() for v in decl.split(",")}
    assert "s_db" in shared
    tail = body[max(body.rfind("__syncthreads()"), body.rfind("__syncwarp()")):]
    assert "__shfl_sync" in tail and "threshold_word" in tail
    written = {v for v in shared if re.search(r"\b" + v + r"(\[[^\]]*\])?\s*=[^=]", tail)}
    assert not written


def test_the_tuner_times_the_launch_that_a_run_makes():
    """Shared memory, kernel and first-unit order of a sweep come from one
    function, for the tuner's timings as for the run: the tuner timed units of
    fewer than 128 words with first units by place, which runs take by index."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "pa_engine.cu")).read())
    setups = [m.start() for m in re.finditer(r"\b(ssc_bits_setup|msc_cluster_setup|sweep_setup)\(", text)]
    one = re.search(r"cudaError_t sweep_grid\(.*?\n  }\n", text, flags=re.S)
    assert one and len(re.findall(r"\bsweep_grid\(", text)) == 3  # itself, the run's launches, the tuner's
    outside = [text[i:i + 60] for i in setups if not one.start() <= i < one.end()]
    assert len(outside) == 1 and outside[0].startswith("msc_cluster_setup(2, 1024")  # an occupancy query
