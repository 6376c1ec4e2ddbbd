"""Order of the converting warps' waits in the grouped GEMMs (hecate_b200/csrc/hmoe_prefill_order.h), walked through on the host: whatever the order of
the items, a stage's wait for codes must not pass on the phase before the one it means."""
import ctypes
import itertools
import os
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include "hmoe_prefill_order.h"
static hmoe::CodeOrder order;
extern "C" void begin() { order = hmoe::CodeOrder(); }
extern "C" int wait_first(int i8) { return order.wait_first(i8 != 0); }
extern "C" int ncode() { return hmoe::PF_NCODE; }
"""


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    src, so = d / "order.cpp", d / "order.so"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "hecate_b200", "csrc"), "-o", str(so), str(src)])
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("stages", [(1, 1, 1, 1), (2, 2, 2, 2), (1, 2, 3, 4), (3, 1, 5, 2), (16, 3, 1, 7)])
def test_every_code_wait_is_behind_the_use_before(order, stages):
    n = order.ncode()
    for i8 in itertools.product((False, True), repeat=len(stages)):
        order.begin()
        owner, t, done = [], 0, 0                                # owner[c] = stage of code c; the codes of stages before `done` are known to be in
        for count, int8 in zip(stages, i8):
            if order.wait_first(int(int8)):
                done = t
            for _ in range(count):
                if int8:
                    done = max(done, t - 1)                      # its operand slot is free: so are the stages up to t - 2
                for _ in range(2 if int8 else 1):
                    if len(owner) >= n:
                        before = owner[len(owner) - n]
                        assert (before - t) % 2 == 0 or before < done, (stages, i8, t)      # waited for by the same group, or known to be in
                    owner.append(t)
                t += 1
