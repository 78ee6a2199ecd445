"""Kernels that may start before the kernel in front of them has ended (float_common.cuh, chain_enter): nothing in their source
may promise that their operands stay as they are while they run, nor read or write before the wait what another kernel touches."""
import glob
import importlib
import os
import re
import threading

import pytest
import torch

from conftest import PKG, ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, PKG, "csrc", "float_*.cu*")))


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _kernels(text):
    """(name, parameters, body) of every __global__ function"""
    for m in re.finditer(r"__global__ void __launch_bounds__\([^\n]*\)\n(\w+)\(", text):
        i = j = m.end()
        depth = 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[j], 0)
            j += 1
        parameters, k = text[i:j - 1], text.index("{", j) + 1
        begin, depth = k, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), parameters, text[begin:k - 1]


CHAINED = {name: (parameters, body) for path in SOURCES for name, parameters, body in _kernels(_code(path)) if "chain_enter()" in body}


def test_every_overlapping_launch_is_of_a_kernel_that_waits():
    launched = {n for path in SOURCES for n in re.findall(r"fp_launch\((\w+_kernel)", _code(path))}
    assert launched and launched == set(CHAINED)


@pytest.mark.parametrize("name", sorted(CHAINED))
def test_operands_of_a_chained_kernel_may_change_while_it_is_resident(name):
    parameters, body = CHAINED[name]
    assert "__restrict__" not in parameters + body


def test_no_load_of_the_chain_goes_through_the_non_coherent_path():
    for path in SOURCES:
        text = _code(path)
        if "chain_enter()" in text:
            assert "ld.global.nc" not in text and "__ldg" not in text and "ld.global.constant" not in text, path


def test_a_thread_records_its_own_calls_only(float_libpath, monkeypatch):
    """another thread's layer is neither recorded nor told that its weights are old"""
    K = importlib.import_module(PKG + ".float_kernel")
    seen = []
    monkeypatch.setattr(K, "_stream", lambda: 0)
    monkeypatch.setattr(K, "_linear", lambda *args: seen.append("plain") or 0)
    monkeypatch.setattr(K, "_linear_early", lambda *args: seen.append("early") or 0)
    A, W, out = torch.zeros(3, 8), torch.zeros(16, 8), torch.zeros(3, 16)
    with K.Recording() as calls:
        other = threading.Thread(target=K.linear, args=(A, W, out))
        other.start()
        other.join()
        assert seen == ["plain"] and not calls.calls and not calls.held
        K.linear(A, W, out)
    K.linear(A, W, out)
    assert seen == ["plain", "early", "plain"] and len(calls.calls) == 1 and calls.held[0] is A
