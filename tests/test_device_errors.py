"""Each code that a kernel can leave in the device error flag has its own message,
and each kind of bounded wait records its own code. Read off the sources: the
grid barrier's limit (over ten seconds) is not run out on a GPU."""

import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "vikalp_b200", "csrc")


def _text(name):
    return open(os.path.join(CSRC, name)).read()


def test_every_device_error_has_its_own_message():
    codes = re.findall(r"(kDevErr\w+) = [1-9]\d*", re.search(r"enum DeviceError[^;]*;", _text("vk_common.cuh")).group())
    assert len(codes) == 2
    report = re.search(r"void check_device_error\(.*?\n}\n", _text("vk_csr.cu"), re.S).group()
    texts = [re.search(c + r'\s*\?\s*"([^"]+)"', report).group(1) for c in codes]
    assert len(set(texts)) == len(codes) and all("timed out" in t for t in texts)


def test_every_wait_records_its_own_code():
    recorded = {name: set(re.findall(r"atomicCAS\([^;]*(kDevErr\w+)", _text(name)))
                for name in ("vk_csr.cuh", "vk_resident.cuh")}
    assert recorded == {"vk_csr.cuh": {"kDevErrBarrierTimeout"}, "vk_resident.cuh": {"kDevErrGridTimeout"}}
