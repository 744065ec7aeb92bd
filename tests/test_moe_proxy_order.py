"""Rows that peers stored are read by TMA only behind a proxy fence (checked in the source: a missing
fence shows on several GPUs only, and there only now and then)."""

import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "lplb_b200" / "csrc" / "moe_gemm.cuh"


def _producer():
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    begin = text.index("warp == 0) {", text.index("__global__"))
    return text[:begin], text[begin : text.index("warp == 1) {", begin)]


def test_the_producer_fences_after_every_acquire_of_a_peers_flag():
    before, producer = _producer()
    # the acquires that a producer's loads depend on: the dispatch flags, polled before the roles
    # start, and the arrival counters of the fused dispatch, polled per expert
    assert before.count("ld.acquire.sys") == 1 and "args.wait_flags + r" in before
    assert producer.count("ld.acquire.sys") == 1 and "args.arrived" in producer
    loop = producer.index("find(t)")
    flags = producer.find("if (args.wait_flags != nullptr) fence_proxy_async_global();")
    assert 0 <= flags < loop, "no fence between the flags' acquire and the first load"
    acquire, first_load = producer.index("ld.acquire.sys"), producer.index("tma_pair_load")
    fence = producer.find("fence_proxy_async_global", acquire)
    assert acquire < fence < first_load, "no fence between an expert's arrival and its loads"
