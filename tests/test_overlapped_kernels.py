"""Kernels launched while the one before them may still run
(cudaLaunchAttributeProgrammaticStreamSerialization): each waits before its
first memory access and promises the compiler nothing about memory that the
kernel before it writes. Read from the source, no GPU needed."""
import os
import re

from conftest import ROOT

SOURCE = open(os.path.join(ROOT, "gyunity_b200", "csrc", "gyt_render.cu")).read()

# written by copies from the host only, which such a launch does not overlap
HOST_WRITTEN = {"list"}


def _kernels():
    """name -> (parameters, body) of every kernel."""
    out = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(k_\w+)\(([^{]*)\)\s*\{", SOURCE):
        out[m.group(1)] = m.group(2), SOURCE[m.end():SOURCE.index("\n}\n", m.end())]
    return out


def _overlapped():
    names = set()
    for m in re.finditer(r"\blaunch_next\(([^;]*);", SOURCE):
        names |= set(re.findall(r"\bk_\w+", m.group(1)))
    for m in re.finditer(r"auto\* const (\w+) =([^;]*);", SOURCE):  # kernels chosen before the launch
        if re.search(r"\blaunch_next\([^;]*\b%s," % m.group(1), SOURCE):
            names |= set(re.findall(r"\bk_\w+", m.group(2)))
    return names - {"k_shade_batch"}  # a batch's choice, launched in stream order


def test_overlapped_kernels_wait_and_promise_nothing():
    kernels, names = _kernels(), _overlapped()
    assert {"k_generate", "k_extend", "k_shade", "k_connect", "k_finish", "k_vshade", "k_grad_adj",
            "k_finish_adj"} <= names
    for name in names:
        params, body = kernels[name]
        statements = [s.strip() for s in re.sub(r"//[^\n]*", "", body).split(";")]
        first = next(s for s in statements if "__shared__" not in s)
        assert first == "chain_start()", name
        read_only = re.findall(r"const [\w ]+\* __restrict__ (\w+)", params)
        assert set(read_only) <= HOST_WRITTEN, (name, read_only)
