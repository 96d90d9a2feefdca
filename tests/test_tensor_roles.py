"""The role code of the tensor-core passes (k_tensor_passes, csrc/tensorpass.cuh) run on the
CPU under chosen schedules (tensor_roles_emu.cpp): one CTA, one warp lagging behind all
others, against the oracle. The waits between the roles have to hold for any speed of any
warp, which a run on a GPU seldom shows. No GPU needed."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "zoda-cu_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"(?m)^#(pragma once|include .*)$", "", f.read())


def span(src, pattern):
    """[start, end) of the top-level definition whose first line matches `pattern`, a
    template line before it included."""
    m = re.search(r"(?m)^(template <[^\n]*>\n)?(?=\S)[^\n]*" + pattern, src)
    assert m, pattern
    depth, i = 0, src.index("{", m.end() - 1)
    while True:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        i += 1
        if depth == 0:
            return m.start(), i + (1 if src[i] == ";" else 0)


def take(src, pattern):
    a, b = span(src, pattern)
    return src[a:b] + "\n"


def drop(src, pattern):
    a, b = span(src, pattern)
    return src[:a] + src[b:]


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    d = tmp_path_factory.mktemp("emu")
    (d / "emu_field.inc").write_text(source("field.cuh"))
    tc, kernel, host = source("tcgen05.cuh"), source("tensorpass.cuh"), source("tensorpass.cu")
    for f in (r"\btp_wait_count\(", r"\btp_store8\(", r"\btp_wait1\("):
        kernel = drop(kernel, f)
    kernel = kernel.replace('asm volatile("fence.proxy.async;" ::: "memory");', "emu_fence();")
    assert "asm" not in kernel
    parts = "namespace zb {\n" + take(tc, r"\bbalanced_digits\(")
    parts += "".join(re.findall(r"(?m)^constexpr uint32_t TC_SWZ[^\n]*\n", tc))
    parts += take(tc, r"\btc_smem_desc\(") + take(tc, r"\btc_idesc_u8s8\(") + "}\n" + kernel + "namespace zb {\n"
    for f in (r"struct Blob\b", r"\bcentered_host\(", r"\bquot_host\(", r"\bput_factor\(", r"\bput_entry\(",
              r"\bplane_sums_below\(", r"\btensor_tables_host\("):
        parts += take(host, f)
    (d / "emu_kernel.inc").write_text(parts + "}\n")
    so = d / "emu.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ftree-vectorize", "-w", "-shared", "-fPIC", "-I", str(d),
                    os.path.join(HERE, "tensor_roles_emu.cpp"), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def run(emu, log_s, seed, lag, cols):
    S = 1 << log_s
    data = O.seeded_input(S, cols, seed=seed)
    out = np.full((2 * S, cols), 0xFFFFFFFF, dtype=np.uint32)
    ptr = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32))
    src = np.ascontiguousarray(data)
    rc = emu.tensor_roles_run(log_s, seed, lag, ptr(src), ptr(out), cols)
    assert rc == 0
    w = min(cols, 8)
    for c0 in range(0, cols - w + 1, max(1, (cols - w) // 15)):  # columns of every operand warp
        want = O.encode_rowmajor(np.ascontiguousarray(data[:, c0:c0 + w]))
        assert np.array_equal(out[:, c0:c0 + w], want), (log_s, lag, c0)


# each of the four operand warps slowest in turn: the end mark must not stand in for its arrival
@pytest.mark.parametrize("log_s,lag", [(11, 0), (11, 3), (12, 1), (12, 2)])
def test_slow_operand_warp(emu, log_s, lag):
    run(emu, log_s, 100 * log_s + lag, emu.tensor_roles_first_operand_warp() + lag, 132)


def test_no_slow_warp(emu):
    run(emu, 11, 7, -1, 260)
