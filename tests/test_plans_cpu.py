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

    def ask(calls, rule="linear_plan_pair"):
        code = ("import json, sys\nfrom fllm_b200.ops._lib import load_cuda\nk = load_cuda(build_if_missing=False)\n"
                f"print(json.dumps([k.{rule}(*c) for c in json.load(sys.stdin)]))")
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


# us on 148 SMs of partial or whole products on CTA pairs by (splits over K, features of a tile)
WIDTHS = {(200, 24576, 4096): {(1, 256): 57.5, (1, 224): 52.9, (1, 192): 49.4, (1, 128): 54.7, (2, 224): 56.3},
          (200, 6144, 4096): {(1, 256): 28.2, (1, 96): 20.3, (1, 128): 20.8, (3, 128): 21.3, (2, 192): 21.3, (3, 256): 22.9},
          (512, 6144, 4096): {(1, 256): 29.4, (1, 224): 26.9, (1, 192): 24.4, (2, 192): 29.6},
          (768, 4096, 4096): {(1, 256): 27.2, (1, 224): 24.8, (1, 192): 22.6, (1, 96): 30.4},
          (1024, 6144, 4096): {(1, 256): 48.2, (1, 224): 43.9, (1, 192): 39.9, (1, 128): 45.9},
          (1024, 4096, 12288): {(1, 256): 73.1, (1, 160): 85.2, (1, 128): 86.1, (1, 192): 97.0},
          (2048, 2048, 2048): {(1, 256): 18.3, (1, 160): 21.1, (1, 192): 22.2, (1, 128): 22.3}}


def test_pairs_take_a_fast_width(plan):
    """Within a twentieth of the fastest measured width and number of splits (the sums are left to the consumer)."""
    got = plan([[t, n, k, 148, WORKSPACE, False, True] for t, n, k in WIDTHS], "linear_plan")
    for (size, times), (splits, width) in zip(WIDTHS.items(), got):
        assert times[splits, width] <= 1.05 * min(times.values()), (size, splits, width)


def test_plan_of_widths_keeps_to_its_limits(plan):
    sizes = [(t, n, k) for t in (1, 128, 129, 200, 256, 700, 2048) for n in (64, 248, 256, 260, 1000, 4096, 24576) for k in (56, 64, 320, 4096, 12288)]
    calls = [[t, n, k, sms, ws, gated, deferred] for t, n, k in sizes for sms in (148, 132) for ws in (0, 65536, 8 << 20, WORKSPACE)
             for gated in (False, True) for deferred in (False, True)]
    for (t, n, k, sms, ws, gated, deferred), (p, width) in zip(calls, plan(calls, "linear_plan")):
        assert 0 <= p <= 8 and 96 <= width <= 256 and width % 32 == 0
        if p:
            assert t > 128 and n >= 256 and n % 8 == 0 and k >= 64
        if p > 1:
            assert not (gated and not deferred) and 65536 + p * t * n * 4 <= ws and p * 4 <= -(-k // 64)


# us of packed 4-bit products by [fp16 form][splits over K]
PACKED = {(64, 24576, 4096): {1: {1: 30.9, 2: 30.2, 3: 30.6, 4: 36.8, 6: 42.5, 8: 52.4}, 0: {1: 38.2, 2: 38.8, 3: 37.6, 8: 53.2}},
          (128, 24576, 4096): {1: {1: 38.0, 2: 41.4, 3: 45.7, 8: 73.9}, 0: {1: 40.9, 2: 43.2, 8: 69.5}},
          (128, 1024, 1024): {1: {1: 9.4, 2: 11.8, 4: 11.5}, 0: {1: 6.9, 2: 8.9, 4: 8.6}},
          (8, 57344, 8192): {1: {1: 91.9, 2: 85.4, 4: 83.5}, 0: {1: 138.9, 2: 125.6, 4: 121.5}},
          (128, 16384, 2048): {1: {1: 15.6, 2: 24.6, 4: 35.1}, 0: {1: 14.0, 2: 23.3, 8: 46.5}},
          (64, 8192, 28672): {1: {1: 90.2, 2: 59.0, 4: 60.8}, 0: {1: 124.8, 2: 70.8, 4: 71.8}},
          (16, 4096, 12288): {1: {1: 37.6, 2: 22.9, 3: 18.6, 4: 17.4, 8: 17.9}, 0: {1: 53.4, 4: 17.5, 8: 18.0}},
          (96, 28672, 4096): {1: {1: 34.0, 2: 41.5, 4: 53.1}, 0: {1: 40.0, 2: 50.4, 8: 82.4}}}


def test_packed_products_take_a_fast_form(plan):
    """Within a tenth of the fastest measured form and number of splits."""
    got = plan([[t, n, k, 148, WORKSPACE - 65536, True] for t, n, k in PACKED], "linear_w4_plan")
    for (size, times), (splits, f16) in zip(PACKED.items(), got):
        assert times[f16][splits] <= 1.1 * min(min(v.values()) for v in times.values()), (size, splits, f16)


def test_plan_of_packed_products_keeps_to_its_limits(plan):
    """Partial sums and fp16 rows that have to fit the workspace together, weights that are not exact in fp16, no workspace at all."""
    calls = [[t, n, k, 148, ws, f16] for t in (1, 16, 17, 97, 128) for n in (8, 136, 1024, 57344) for k in (64, 320, 4096, 28672)
             for ws in (0, 4096, 1 << 20, 8 << 20, WORKSPACE) for f16 in (False, True)]
    for (t, n, k, sms, ws, f16), (splits, form) in zip(calls, plan(calls, "linear_w4_plan")):
        rows = (t * k * 2 + t * 4 + 255) // 256 * 256 + 256
        assert 1 <= splits <= 8 and splits <= -(-k // 256) and form <= f16
        assert (splits * t * n * 4 if splits > 1 else 0) + (rows if form else 0) <= ws
