"""Which barriers the kernels signal in another CTA without a release. An arrive without one orders no ordinary memory, so it may only
announce finished tensor-memory operations; shared memory that is handed to (or back to) another CTA needs the releasing form.
Read from the sources: a missing release cannot be shown by running a kernel."""

import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).resolve().parents[1] / "euhedral_b200" / "csrc").glob("*.cu*"))
TENSOR_MEMORY = {"scaled", "acc_empty"}   # scales stored to tensor memory; sums read out of it


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("path", SOURCES, ids=lambda path: path.name)
def test_signals_without_release_announce_tensor_memory_only(path):
    text = code(path)
    barriers = set(re.findall(r"signal_rank_relaxed\(&?(\w+)", text)) - {"uint64_t"}
    assert barriers <= TENSOR_MEMORY, barriers
    # one place issues the relaxed arrive; everything else goes through the two named functions
    assert text.count("mbarrier.arrive.relaxed") == (1 if path.name == "nvfp4_native.cuh" else 0)


def test_the_q3_terms_are_released_to_the_even_cta():
    text = code(next(path for path in SOURCES if path.name == "q3_prefill.cuh"))
    assert "signal_rank(&made[stage], 0u)" in text and "mbar_wait_cluster_or_fail(&made[" in text
    native = code(next(path for path in SOURCES if path.name == "nvfp4_native.cuh"))
    assert native.count("mbarrier.arrive.release.cluster") == 1


def test_the_exchange_buffers_are_released_after_they_were_read():
    text = code(next(path for path in SOURCES if path.name == "nvfp4_decode.cuh"))
    assert "signal_rank(&gather_empty[" in text and "mbar_wait_cluster_or_fail(&gather_empty[" in text
    assert "mbar_wait_cluster_or_fail(&gather_full[" in text   # what the other CTAs' st.async wrote
