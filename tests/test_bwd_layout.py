"""Shared memory of the per-chunk backward kernel: each of its two groups of warps lays its memory out anew when it goes
from mild to steep chunks, at a time of its own.  The tensor memory's address, which both groups read, lies in neither."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rwkv_infctx_trainer_b200", "csrc",
                      "wkv56_chunked_bwd.cu")


def test_the_tensor_memory_address_is_in_no_group_s_memory():
    with open(SOURCE) as f:
        text = f.read()
    for name in ("MildSmem", "SteepSmem"):
        body = re.search(r"struct %s \{(.*?)\n\};" % name, text, re.S).group(1)
        assert "tmem" not in body, name
    assert re.search(r"tmem_base = reinterpret_cast<uint32_t \*>\(smem_raw \+ BWD_GROUPS \* BWD_SMEM\)", text)
    assert re.search(r"smem = BWD_SMEM \* BWD_GROUPS \+ 16;", text)
