"""Waits inside kernels that gave up reach the host (csrc/wait_report.h): the word's count, its one refusal per news, and the engine that asks.  No
kernel is made to wait in vain: the device's part, a count in host memory, is written by the host."""
import os
import re
import subprocess
from collections import deque
from types import SimpleNamespace

import numpy as np
import pytest

from nanovllm import _native as nat

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nano-vllm_b200", "csrc")

PROGRAM = r"""
#include "wait_report.h"
#include <cstdio>
int main() {
    B200WaitReport r;
    uint32_t word = 0;
    auto say = [&](bool times_two = false) {
        std::printf("%u ", r.count());
        for (int i = 0; i <= times_two; ++i) std::printf("%d ", (int)r.news());
    };
    say();            // no launch yet
    r.word = &word;
    say();            // nothing happened
    word += 2;        // as two blocks would
    say(true);
    word += 1;
    say(true);
}
"""


def test_news_is_told_once(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "0", "0", "2", "1", "0", "3", "1", "0"]


def test_libraries_count_and_name_the_error():
    assert nat.load().b200_wait_timeouts() == 0 and nat.load_mix().b200m_wait_timeouts() == 0 and nat.wait_timeouts() == 0
    assert b"gave up" in nat.load().b200_strerror(-7)
    with pytest.raises(nat.WaitTimeout, match="gave up"):
        nat.check_mix(-7)
    with pytest.raises(nat.WaitTimeout, match="gave up"):
        nat.check(-7)


def test_collect_raises_once_per_news(monkeypatch):
    from nanovllm.engine.model_runner import ModelRunner
    run = ModelRunner.__new__(ModelRunner)
    run._done = [SimpleNamespace(synchronize=lambda: None)] * 2
    run.h_err = [[0], [0]]
    run.h_tokens_np = [np.arange(4), np.arange(4)]
    run._waits_seen = 0
    run._pending = deque([(0, 2), (1, 2), (0, 2)])
    count = [0]
    monkeypatch.setattr(nat, "wait_timeouts", lambda: count[0])
    assert run.collect() == [0, 1]
    count[0] = 3
    with pytest.raises(nat.WaitTimeout):
        run.collect()
    assert run.collect() == [0, 1]


def test_every_bounded_wait_reports_and_is_the_whole_warps():
    """A bounded wait has no other sink than the launch's host word, and the warp votes before it answers; lanes answer for themselves in the prompt
    kernel's product warps alone."""
    text = open(os.path.join(CSRC, "tc_common.cuh")).read()
    body = text[text.index("bool bounded_wait_as("):]
    body = body[:body.index("\n}\n")]
    assert body.count("return true") == body.count("if (WHOLE ? __all_sync(0xffffffffu, ok) : ok) return true") == 2
    calls = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")) and name != "tc_common.cuh":
            source = open(os.path.join(CSRC, name)).read()
            calls += source.count("bounded_wait(")
            assert source.count("bounded_wait_as<false>(") == (name == "fa_tc.cuh"), name
            assert source.count("bounded_wait(") == len(re.findall(r"bounded_wait\([^;]*?, dead, p\.report\)", source)), name
    assert calls >= 10
