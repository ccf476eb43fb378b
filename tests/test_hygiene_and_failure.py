"""Source hygiene greps and host-side failure-detection units (no GPU is ever faulted or hung)."""
import os
import re
import time

import pytest

from tah_b200.utils.failure import RankFailure, RankHeartbeat, StepTimeout, StepWatchdog

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _sources(exts=(".py", ".cu", ".cuh", ".h")):
    for base in ("tah_b200", "csrc", "script", "bench.py", "__graft_entry__.py"):
        p = os.path.join(ROOT, base)
        if os.path.isfile(p):
            yield p
            continue
        for d, _, files in os.walk(p):
            for f in files:
                if f.endswith(exts):
                    yield os.path.join(d, f)


def test_no_cluster_multicast_no_triton_no_disassembly():
    bad = []
    # the qualifier this test looks for is assembled from pieces so that this file does not name it
    multicast = "".join([".", "multi", "cast", "::", "clus", "ter"])
    bulk_copy = "".join(["cp", ".", "as", "ync"])
    for path in _sources():
        text = open(path, encoding="utf-8", errors="ignore").read()
        if multicast in text and not path.endswith("comm.cu") and not path.endswith("common.cuh"):
            bad.append((path, "cluster multicast"))
        if multicast in text:
            # even the files that mention the rule must not contain a multicast instruction
            for line in text.splitlines():
                if multicast in line and (bulk_copy in line or "asm" in line):
                    bad.append((path, "multicast instruction"))
        if re.search(r"^\s*(import triton|from triton)", text, re.M):
            bad.append((path, "triton"))
        if re.search(r"cuobjdump|nvdisasm|objdump\s+-d", text):
            bad.append((path, "disassembly tool"))
        if "torch.compile(" in text:
            bad.append((path, "torch.compile"))
        if re.search(r"cu(da)?Memcpy(3D)?Batch" + "Async", text):
            bad.append((path, "closed batched-copy call"))
    assert not bad, bad


def test_every_device_wait_is_bounded():
    """Every spin in the kernels goes through a helper with a time limit."""
    for name in ("gemm_tcgen05.cu", "attn_decode.cu", "attn_prefill.cu", "attn_window.cu", "mlstm.cu"):
        text = open(os.path.join(ROOT, "csrc", name)).read()
        assert "mbar_try_wait(" not in text            # only the bounded mbar_wait() may be called from kernels
        assert "while (true)" not in text and "while(1)" not in text
    for name in ("comm.cu", "optim.cu"):
        text = open(os.path.join(ROOT, "csrc", name)).read()
        assert "WAIT_TIMEOUT_NS" in text and "STATUS_TIMEOUT_PEER_FLAG" in text


def test_waits_of_the_persistent_backward_and_few_token_kernels_are_bounded():
    """The same for the persistent product, the attention backward and the one wait of the fused few-token product."""
    for name in ("gemm_persist.cu", "attn_prefill_bwd.cu"):
        text = open(os.path.join(ROOT, "csrc", name)).read()
        assert "mbar_try_wait(" not in text and "while (true)" not in text and "while(1)" not in text
    text = open(os.path.join(ROOT, "csrc", "gemm_few.cu")).read()
    assert text.count("ld_acquire(p.sync)") == text.count("now - t0 > WAIT_TIMEOUT_NS") == 1


# operands that are constants of a chain of launches: weights and tables
_CONSTANTS = {"w", "A", "E", "b", "freq", "w_in", "act", "dot_w", "dot_b"}


def _balanced(text, i, opening, closing):
    depth = 1
    while depth:
        depth += (text[i] == opening) - (text[i] == closing)
        i += 1
    return i


def test_kernels_that_start_early_read_what_was_written_before_through_plain_pointers():
    """A kernel that waits for the launch before it (pdl_wait) has ``__restrict__`` on weights and tables alone: what is read or written through
    such a pointer may move ahead of the wait."""
    seen, bad = 0, []
    for path in _sources((".cu", ".cuh")):
        text = open(path, encoding="utf-8").read()
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^()]*(?:\([^()]*\)[^()]*)*\)\s*)?(\w+)\s*\(", text):
            end = _balanced(text, m.end(), "(", ")")
            body = re.compile(r"[{;]").search(text, end).start()
            if text[body] == "{" and "pdl_wait()" in text[body:_balanced(text, body + 1, "{", "}")]:
                seen += 1
                bad += [(m.group(1), n) for n in re.findall(r"__restrict__\s+(\w+)", text[m.end():end]) if n not in _CONSTANTS]
    assert seen > 20 and not bad, bad


class _DictStore(dict):
    def set(self, k, v):
        self[k] = v

    def get(self, k):
        return self[k]


def test_heartbeat_with_fake_store():
    store = _DictStore()
    a = RankHeartbeat(store, 0, 2, interval_s=0.05).start()
    b = RankHeartbeat(store, 1, 2, interval_s=0.05).start()
    time.sleep(0.2)
    a.check_peers(timeout_s=0.3)
    b.stop()                                             # rank 1 "dies": its counter stops moving
    with pytest.raises(RankFailure) as info:
        t0 = time.time()
        while time.time() - t0 < 3:
            a.check_peers(timeout_s=0.3)
            time.sleep(0.05)
    assert info.value.dead == [1]
    a.stop()


def test_heartbeat_missing_key_counts_as_dead():
    store = _DictStore()
    a = RankHeartbeat(store, 0, 2, interval_s=0.05)
    a.beat()
    a.check_peers(timeout_s=0.1)                         # first look only records
    time.sleep(0.2)
    with pytest.raises(RankFailure):
        a.check_peers(timeout_s=0.1)


def test_step_watchdog():
    with StepWatchdog(1.0):
        pass
    with pytest.raises(StepTimeout):
        with StepWatchdog(0.05):
            time.sleep(0.2)
    fired = []
    with StepWatchdog(0.05, on_timeout=lambda: fired.append(1)):
        time.sleep(0.2)
    assert fired == [1]
