"""The rules that pick one form of a kernel or another by size alone (csrc/rules.h), compiled for the host and checked at
the sizes where each form was measured to be the faster one. 148 SMs throughout."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148

_WRAPPERS = """
#include "rules.h"
extern "C" bool attn_lone(long long items, int sms) { return b200ait::attn_lone(items, sms); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    work = tmp_path_factory.mktemp("rules")
    src, lib = work / "rules.cpp", work / "rules.so"
    src.write_text(_WRAPPERS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "aitemplate_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    lib = ctypes.CDLL(str(lib))
    lib.attn_lone.restype = ctypes.c_bool
    return lib


@pytest.mark.parametrize("items,lone", [(1, True), (16, True), (128, True), (148, True), (149, False), (296, False)])
def test_wide_heads_with_an_item_per_sm_keep_four_stages(rules, items, lone):
    assert rules.attn_lone(ctypes.c_longlong(items), SMS) == lone
