"""The benchmark's traffic figures: each names a capture that is there, is of the
kernel that the benchmark names beside it, and follows from the capture's DRAM
bytes (mean of the proton and electron launches over 4,096 tracers; the captures
give whole megabytes, so 0.5 of the smallest launch's 69: 1 %)."""
import os
import re

import pytest

from conftest import ROOT


def _bench():
    with open(os.path.join(ROOT, "bench.py")) as f:
        return f.read()


def test_every_named_profile_is_there():
    named = re.findall(r"profiles/[\w*.]+", _bench())
    assert named and all(os.path.exists(os.path.join(ROOT, p)) for p in named), named


@pytest.mark.parametrize("key,kernel", [("steps", "steps_packed_kernel"), ("plain_steps", "plain_steps_kernel")])
def test_traffic_follows_from_the_capture(key, kernel):
    text = _bench()
    const = {"steps": "STEPS_PROFILE", "plain_steps": "PLAIN_PROFILE"}[key]
    scope = {}
    for line in re.findall(r"^(?:STEPS_PROFILE|NCU_DRAM_BYTES_PER_TRACER)\b.*$", text, re.M):
        exec(line, scope)
    assert f'"kernel": "{kernel}' in text
    with open(os.path.join(ROOT, scope[const])) as f:
        capture = f.read()
    launches = re.findall(r"kernel: (\w+)<.*?DRAM read / write\s+(\d+) / (\d+) MB", capture, re.S)
    assert len(launches) == 2 and all(k == kernel for k, _, _ in launches) and "4,096 tracers" in capture
    mean = sum(float(r) + float(w) for _, r, w in launches) * 1e6 / 2 / 4096
    assert abs(scope["NCU_DRAM_BYTES_PER_TRACER"][key] / mean - 1) <= 0.01
