"""The C-ABI library loads without a GPU and exports every symbol the public
header declares; the Python loader's signature table covers the same set."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def header_symbols():
    src = open(os.path.join(ROOT, "include", "tlb200.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(tlb_[a-z0-9_]+)\s*\(", src)))


def test_library_exports_every_declared_symbol():
    from cpp_tensorlib_b200 import _lib
    L = ctypes.CDLL(_lib.LIB_PATH)
    names = header_symbols()
    assert len(names) >= 30
    for n in names:
        assert hasattr(L, n), f"{n} declared in include/tlb200.h but not exported"
    assert sorted(_lib.SIGNATURES) == names


def test_no_compute_without_gpu_fails_loudly():
    import torch
    if torch.cuda.is_available():
        pytest.skip("GPU present")
    from cpp_tensorlib_b200 import TlbError, check, lib
    assert lib().tlb_device_count() == 0
    with pytest.raises(TlbError):
        check(lib().tlb_init(0))
    assert lib().tlb_q4_bytes(4864, 896) == 2179072 + 544768  # include/types.h:29-31


@pytest.mark.parametrize("name", ["gemm_q4_tc.cu", "gemm_q4_tc2.cu", "gemm_bf16_tc.cu", "attn_decode_mma.cu",
                                  "attn_prefill_mma.cu", "attn_prefill_bf16.cu"])
def test_whole_warps_agree_on_a_wait(name):
    """A wait that gives up for some lanes of a warp and not for others leaves them at different barriers.  Where whole
    warps wait, in front of warp-wide instructions, they vote (mbar_wait_warp) or go on whatever the outcome; a branch on
    a plain wait is for a single lane."""
    text = open(os.path.join(ROOT, "cpp_tensorlib_b200", "csrc", name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    heads, start, single = [], 0, 0
    for i, ch in enumerate(text):
        if ch in "{};":
            if "mbar_wait_bounded(" in text[start:i] and not re.search(r"if \((\w+)\) \1 = mbar_wait_bounded\(", text[start:i]):
                assert any("lane == 0" in h or "producer" in h for h in heads), text[start:i].strip()
                single += 1
            if ch == "{":
                heads.append(text[start:i])
            elif ch == "}":
                heads.pop()
            start = i + 1
    assert single or name == "attn_prefill_bf16.cu"
