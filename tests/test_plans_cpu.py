"""Rules of dispatch that are decided on the host: which form of a kernel takes a product."""
import json
import subprocess
import sys

import pytest

from fllm_b200._build import LIB_CUDA, ROOT

WORKSPACE = 96 << 20

# us on 148 SMs, (one-CTA tiles, CTA pairs), of products whose sums are added by a kernel of their own
MEASURED = {(129, 512, 512): (7.12, 12.49), (200, 2048, 2048): (9.99, 15.44), (512, 3072, 2048): (14.53, 22.11), (1024, 2048, 2048): (15.07, 17.48),
            (2048, 1000, 320): (7.16, 8.70), (256, 256, 4096): (9.10, 15.02), (512, 768, 3072): (12.16, 20.11), (300, 24576, 4096): (67.79, 71.77),
            (256, 6144, 4096): (24.40, 28.79), (1024, 1024, 1024): (10.38, 12.03),
            (200, 24576, 4096): (66.07, 54.95), (300, 4096, 12288): (59.46, 45.12), (512, 6144, 4096): (41.24, 29.33), (768, 4096, 4096): (42.06, 28.66),
            (1024, 2048, 8192): (41.96, 36.79), (1536, 2048, 2048): (24.25, 18.00), (2048, 24576, 4096): (313.67, 268.59), (1024, 3072, 2048): (24.75, 19.59),
            (200, 16384, 2048): (24.47, 20.94), (2048, 768, 3072): (18.74, 24.12)}


@pytest.fixture(scope="module")
def plan():
    """The rule of the built library, asked in a process of its own (a CPU test loads no kernels)."""
    if not LIB_CUDA.exists():
        pytest.skip("the CUDA library is not built")

    def ask(calls):
        code = ("import json, sys\nfrom fllm_b200.ops._lib import load_cuda\nk = load_cuda(build_if_missing=False)\n"
                "print(json.dumps([k.linear_plan_pair(*c) for c in json.load(sys.stdin)]))")
        out = subprocess.run([sys.executable, "-c", code], input=json.dumps(calls), capture_output=True, text=True, check=True, cwd=ROOT.parent, timeout=300)
        return json.loads(out.stdout.splitlines()[-1])
    return ask


def test_products_take_the_faster_form(plan):
    got = plan([[t, n, k, 148, WORKSPACE, False, False] for t, n, k in MEASURED])
    assert {s: p > 0 for s, p in zip(MEASURED, got)} == {s: pair < one for s, (one, pair) in MEASURED.items()}


def test_plan_of_pairs_keeps_to_its_limits(plan):
    """What the pair kernel does not take, sums that have to be whole, and partial sums that have to fit the workspace."""
    sizes = [(t, n, k) for t in (1, 128, 129, 200, 256, 700, 2048) for n in (64, 248, 256, 260, 1000, 4096, 24576) for k in (56, 64, 320, 4096, 12288)]
    calls = [[t, n, k, sms, ws, gated, deferred] for t, n, k in sizes for sms in (148, 132) for ws in (0, 65536, 8 << 20, WORKSPACE)
             for gated in (False, True) for deferred in (False, True)]
    for (t, n, k, sms, ws, gated, deferred), p in zip(calls, plan(calls)):
        assert 0 <= p <= 8
        if p:
            assert t > 128 and n >= 256 and n % 8 == 0 and k >= 64
        if p > 1:
            assert not (gated and not deferred) and 65536 + p * t * n * 4 <= ws and p * 4 <= -(-k // 64)
