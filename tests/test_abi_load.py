"""CPU: the C-ABI library loads and exports every symbol include/spyb.h declares; host-only calls behave."""
import ctypes as C
import os

import pytest

from spy_b200 import backend
from spy_b200 import quants


def test_library_exports_every_declared_symbol():
    if not os.path.exists(backend.LIB_PATH):
        import __graft_entry__
        __graft_entry__.build()
    l = C.CDLL(backend.LIB_PATH)
    declared = backend.exported_symbols()
    assert len(declared) >= 20
    missing = [s for s in declared if not hasattr(l, s)]
    assert not missing, f"declared in spyb.h but not exported: {missing}"


def test_is_support_matches_the_operator_table():
    l = backend.lib()
    for name, op in backend.OP.items():
        assert l.spyb_is_support(op) == 1, name
    for op in (6, 7, 12, 14, 15, 16, 19, 21, 22, 24, 25, 28):   # MaskedCopy .. Quantize: not on the LLaMa path
        assert l.spyb_is_support(op) == 0


def test_create_fails_loudly_without_a_gpu():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    with pytest.raises(backend.SpybError):
        backend.B200Backend(0)


def test_shared_memory_ledger_is_kept_per_device_and_kernel():
    """cudaFuncAttributeMaxDynamicSharedMemorySize belongs to a (device, kernel) pair: the library's record of what it
    has already raised must be kept per pair, or the second device of a process never gets the attribute set."""
    assert backend.lib().spyb_selftest_host() == 0


def test_attention_ring_slots_keep_their_warps():
    """The ring of the long-context attention kernel, for all contexts and numbers of CTAs: a slot's successive stages come from one copy warp
    and go to one reader, or a wait by parity could take a phase for the one two before it (stages overwritten while they are read, or a
    wait that never ends)."""
    assert backend.lib().spyb_selftest_host() == 0


@pytest.mark.parametrize("rows,k,tokens,form", [
    # measured on 148 SMs, us with tiles of 16 / 8 tokens by one CTA, 16 / 8 by two
    (22148, 1728, 5, (8, 1)),       # 22.3 / 17.0 / 25.0 / 20.1
    (1548, 2304, 58, (8, 1)),       # 16.2 / 12.7 / 14.0 / 17.8
    (10192, 1088, 54, (8, 1)),      # 22.5 / 20.7 / 29.7 / 32.5
    (4140, 2464, 23, (8, 1)),       # 16.7 / 13.2 / 14.7 / 18.5
    (1680, 2208, 79, (8, 1)),       # 15.6 / 13.3 / 16.2 / 18.8
    (8348, 4160, 12, (16, 2)),      # 25.8 / 22.5 / 19.7 / 28.5
    (4096, 11008, 8, (8, 2)),       # 59.2 / 51.3 / 38.2 / 33.9
    (7560, 5792, 15, (16, 2)),      # 34.4 / 32.1 / 24.3 / 38.4
    (22016, 4096, 448, (16, 1)),    # 655 / 993 / 826 / 1185
    (32000, 4096, 16, (16, 1)),     # 54.7 / 82.7 / 63.1 / 85.3
])
def test_prompt_gemm_takes_the_form_that_measures_fastest(rows, k, tokens, form):
    tok, ctas = C.c_int32(0), C.c_int32(0)
    assert backend.lib().spyb_prefill_form(rows, k, tokens, 148, C.byref(tok), C.byref(ctas)) == backend.SUCCESS
    assert (tok.value, ctas.value) == form


@pytest.mark.parametrize("qt,rows,k,tokens,shared", [
    # measured on 148 SMs, us a submit with whole / shared last tiles, from one backend and from three in turn
    (quants.Q4_0, 12288, 4096, 21, True),      # 45.9 / 37.2, 37.6 / 34.2
    (quants.Q4_0, 32000, 4096, 16, False),     # 52.5 / 52.7, 45.2 / 49.8
    (quants.Q4_0, 5120, 13824, 32, False),     # 70.9 / 57.7, 40.4 / 54.2
    (quants.Q6_K, 6520, 6144, 39, False),      # 32.6 / 31.9, 21.8 / 26.8
    (quants.Q4_K, 11008, 4096, 64, True),      # 45.4 / 32.5, 28.5 / 29.7
    (quants.Q4_K, 4096, 4096, 512, True),      # 79.0 / 72.9, 73.7 / 70.3
])
def test_operators_share_tiles_where_that_pays_beside_others_too(qt, rows, k, tokens, shared):
    assert (backend.prefill_plan(qt, rows, k, tokens)[2] == 2) == shared


def test_uploads_have_arrived_when_they_return():
    """A plain cudaMemcpy from pageable memory may return before its last piece has arrived, and a non-blocking stream does not wait for the legacy one: what
    the legacy stream copies or clears is waited for beside the call."""
    csrc = os.path.join(os.path.dirname(backend.__file__), "csrc")
    for name in sorted(os.listdir(csrc)):
        if name.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(csrc, name)) as f:
                lines = f.read().split("\n")
            for i, line in enumerate(lines):
                if "cudaMemset(" in line or ("cudaMemcpy(" in line and "HostToDevice" in line):
                    assert "cudaStreamSynchronize(cudaStreamLegacy)" in line + lines[i + 1], (name, line)
