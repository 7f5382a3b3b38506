"""A pass whose kernels left an error fails, also when another caller has read and cleared the device's word since: the host's part with g++, and a step of a
decoder on a device whose word another model has set."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import jasmine_b200 as jb

CSRC = Path(__file__).resolve().parents[1] / "jasmine_b200" / "csrc"

PROGRAM = r"""
#include "pass_errors.h"
enum Status { OK = 0, FROM_WORD = 1, FROM_COPY = 2 };
int checks = 0, failed_with = 0;
Status run(std::initializer_list<int32_t> words, Status word) {
    checks = failed_with = 0;
    return jsm::pass_status(words.begin(), (int)words.size(), [&] { ++checks; return word; }, [&](int code) { failed_with = code; return FROM_COPY; });
}
int main() {
    if (run({0, 0, 0}, FROM_WORD) != OK || checks != 0) return 1;        // nothing in the copies: the word is not asked
    if (run({}, FROM_WORD) != OK) return 2;
    if (run({0, 7, 0}, FROM_WORD) != FROM_WORD || checks != 1 || failed_with != 0) return 3;
    if (run({0, 0, 7}, OK) != FROM_COPY || checks != 1 || failed_with != 7) return 4;  // somebody has cleared the word
    if (run({-3, 7}, OK) != FROM_COPY || failed_with != -3) return 5;
    return 0;
}
"""


def test_a_code_that_was_seen_is_not_dropped(tmp_path):
    src, exe = tmp_path / "errors.cpp", tmp_path / "errors"
    src.write_text("#include <initializer_list>\n" + PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


@pytest.mark.gpu
def test_a_step_reports_the_word_and_clears_it():
    import torch
    import zugolorn_oracle as zo
    import zugolorn_util as zu
    from jasmine_b200.model import Llama
    cfg = zu.config([zu.mamba()])
    w = zu.random_weights(cfg, 1)
    toks = zu.tokens(6, cfg["vocab"], 2)
    want = zo.forward(cfg, zu.oracle_weights(w), toks[:4])[3:]
    m = zu.build(cfg, w)
    m.step([(m.open(), toks[:3])], [2])
    other = Llama(1, 256, 2, 2, 512, 1024, max_batch=1, max_context=64)
    ids = torch.zeros(64, dtype=torch.int32, device="cuda")
    other.prefill(ids, 0, ids[:1])
    other.decode_step(ids[:1], ids[1:2])  # a context overflow: the device's word is set, and nobody has read it
    torch.cuda.synchronize()
    nxt, lg = np.empty(1, np.int32), np.empty((1, cfg["vocab"]), np.float32)
    with pytest.raises(jb.JsmError) as e:
        m.step_active(np.array(toks[3:4], np.int32), nxt, lg)
    assert e.value.status == jb.SHAPE
    jb.check_device_errors()  # (cleared)
    row = m.open()
    m.step([(row, toks[:3])], [2])
    _, lg = m.step([(row, toks[3:4])], [0])
    assert zu.error(lg, want) < 4e-5  # (the bar of the other fp32 models)
    m.close()
    other.close()
