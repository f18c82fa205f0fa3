"""Reads of asynchronous results in the tensor-core batched kernel's source.

What a tensor-memory load writes may not be touched before the wait that
completes it.  Code that breaks this can give right answers for as long as the
assembler happens to order it, so the source itself is checked.
"""
import os
import re

import entropydecreaseboltzmann_gb300

SOURCE = os.path.join(os.path.dirname(entropydecreaseboltzmann_gb300.__file__), "csrc",
                      "edb_kernels_calqtc.cu")


def _text():
    with open(SOURCE) as f:
        return f.read()


def _asm(text):
    """The instruction text of every asm statement."""
    blocks = re.findall(r"asm(?: volatile)?\(\s*((?:\"(?:[^\"\\\\]|\\\\.)*\"\s*)+)", text)
    return ["".join(re.findall(r"\"((?:[^\"\\\\]|\\\\.)*)\"", b)) for b in blocks]


def test_a_tensor_memory_load_stands_alone_in_its_asm_statement():
    loads = [a for a in _asm(_text()) if "tcgen05.ld" in a]
    assert len(loads) == 2
    for a in loads:
        assert a.count(";") == 1 and "mov" not in a, a


def test_the_read_ahead_of_the_last_step_is_completed():
    # the read ahead always fills x[0]: nothing of the fold, which ends the
    # last step, comes before its wait
    fold = _text().split("if (--fc == 0 || i + 1 == total) {")
    assert len(fold) == 2
    code = re.sub(r"//[^\n]*", "", fold[1])
    assert re.match(r"\s*fc = a\.FL;\s*tc_wait_ld\(x\[0\]\);", code)


def test_one_lane_gives_shared_memory_back_only_after_the_whole_warp():
    # BE: a stage of weights, PE: a staged plane; both are read by all lanes
    releases = re.findall(r"([^\n]*)\n\s*mbar_arrive\(bar\((?:BE|PE) ", _text())
    assert len(releases) == 2
    for line in releases:
        assert line.strip() == "__syncwarp();", line


def test_the_drain_after_a_wait_ran_out_has_one_limit_and_its_outcome_counts():
    csrc = os.path.dirname(SOURCE)
    limits = []
    for name in sorted(os.listdir(csrc)):
        with open(os.path.join(csrc, name)) as f:
            limits += re.findall(r"constexpr unsigned long long (\w*DRAIN\w*) = (\d+)ull;", f.read())
    assert limits == [("DRAIN_LIMIT_NS", "1000000000")]
    # matrix products still in flight: the launch reports it
    assert "if (!mbar_poll(bar(XD), 0, DRAIN_LIMIT_NS)) lim = 0;" in _text()
