"""Launches behind another stream's event are ordinary ones: programmatic
serialization orders a kernel after the one before it on its own stream, so
wherever a stream that kernels are launched on waits for another stream, the
wait goes through Impl::wait_for, which takes the early start from the next
launch.  Read from the source: on the device the early start shows only as a
rare overwrite of a copy still in flight."""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "kami-hair-solver_gb300" / "csrc" / "khs_engine.cu"


def test_cross_stream_waits_make_the_next_launch_ordinary():
    text = SOURCE.read_text()
    helper = re.search(r"void wait_for\(cudaStream_t s, cudaEvent_t e\)\s*\{(.*?)\}", text, re.S)
    assert helper and "ordinary = s;" in helper.group(1)
    waits = re.findall(r"cudaStreamWaitEvent\((.*?),", text)
    assert waits.count("s") == 1  # wait_for itself
    # The copy stream carries copies only, no kernels.
    assert [w for w in waits if w != "s"] == ["I.copy_stream"] * (len(waits) - 1)
    assert not re.search(r"(launch_on|start)\([^)]*copy_stream", text)
