"""Rules of the kernels that no run can show to hold, since a GPU that happens to keep them behaves alike: checked in the source."""
import glob
import os
import re


def test_barriers_are_polled_once_only_by_whole_warps(t0):
    # Whether a phase is over may be answered differently lane by lane.  A wait asks until every lane has the same answer; a single look whose answer decides
    # where a warp goes has to be voted on, inside the helper, so that no kernel calls the instruction or an unvoted helper itself.
    csrc = os.path.join(os.path.dirname(os.path.dirname(t0.HEADER_PATH)), "rust-gpu_b200", "csrc")
    for path in sorted(glob.glob(os.path.join(csrc, "*.cu"))):
        text = open(path).read()
        assert not re.search(r"mbarrier\.(test|try)_wait|mbar_(test|try)_wait\(", text), path
    helpers = open(os.path.join(csrc, "ptx_sm100.cuh")).read()
    looks = re.findall(r"__device__ __forceinline__ bool (\w+)\([^)]*\) \{\n(.*?)\n\}", helpers, flags=re.S)
    single = [(name, body) for name, body in looks if "mbarrier.test_wait" in body]
    assert single and all("return __all_sync(0xFFFFFFFFu" in body for _, body in single), [name for name, _ in single]


def test_the_streaming_epilogue_follows_no_ring(t0):
    # A wait asks for a parity, which every second phase of a barrier answers: a role may wait on a ring's barrier only if it waits for every phase.  The epilogue
    # warps of the streaming kernel come by once per piece of a range.
    csrc = os.path.join(os.path.dirname(os.path.dirname(t0.HEADER_PATH)), "rust-gpu_b200", "csrc")
    text = open(os.path.join(csrc, "w4a16_stream.cu")).read()
    role = text[text.index("four warps: accumulators to y"):text.index("give copies and UMMAs already in flight")]
    waits = re.findall(r"mbar_wait\w*\((\w+)", role)
    assert sorted(set(waits)) == ["acc_full", "end_near"], waits
