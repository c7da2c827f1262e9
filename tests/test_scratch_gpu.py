"""GPU tests of what the library keeps of the device's memory for operands it prepares
(A transposed, rows copied): bounded, and given back.  The reference allocates
nothing (src/sgemm.cuh:19-48)."""
import pytest

import oracle
import sgemm_b200 as sg

pytestmark = pytest.mark.gpu

KEPT = 4 << 30  # bytes the scratch pool keeps between calls, and all plans hold
PER_CALL = 1 << 30
GRAIN = 64 << 20  # the driver's allocation granularity, with room


def _reserved():
    import torch

    torch.cuda.synchronize()  # unused memory beyond the bound goes back here
    return sg.pool_usage()[1]


def test_a_call_keeps_no_more_than_its_share():
    import torch

    before = _reserved()
    m, n, k = 20000, 2048, 20000  # A transposed would be 1.6 GB
    A, B = torch.empty((m, k), device="cuda"), torch.empty((k, n), device="cuda")
    C = torch.zeros((m, n), device="cuda")
    sg.fill_random(A, 61, 1, sg.DIST_UNIFORM_PM1)
    sg.fill_random(B, 61, 2, sg.DIST_UNIFORM_PM1)
    for _ in range(2):
        sg.sgemm(A, B, C)
    assert _reserved() <= before + PER_CALL + GRAIN
    rows = [0, 77, m - 1]
    want = oracle.sgemm_basic(A[rows].cpu().numpy(), B.cpu().numpy(),
                              C[rows].cpu().numpy(), 1.0, 0.0, basic=False)
    assert (C[rows].cpu().numpy() == want).all()
    assert sg.device_status() == sg.OK


def test_plans_hold_a_bounded_share_of_the_device():
    import torch

    _reserved()
    used0, reserved0 = sg.pool_usage()
    side = 25600  # two copies of A are over the plans' share
    A = torch.empty((side, side), device="cuda")
    B, C = torch.zeros((side, 512), device="cuda"), torch.zeros((side, 512), device="cuda")
    one = sg.GroupedPlan([(A, B, C, 1.0, 0.0)])
    used1 = sg.pool_usage()[0]
    assert used1 - used0 >= 4 * side * side  # the first copy fits
    two = sg.GroupedPlan([(A, B, C, 1.0, 0.0), (A[:1000], B, C[:1000], 1.0, 0.0)])
    used2 = sg.pool_usage()[0]
    assert used2 - used0 <= KEPT + GRAIN
    assert used2 - used1 >= 4 * 1000 * side  # what still fits is prepared
    one.close()
    two.close()
    _reserved()
    used3, reserved3 = sg.pool_usage()
    assert used3 == used0
    assert reserved3 <= max(reserved0, KEPT) + GRAIN
    again = sg.GroupedPlan([(A, B, C, 1.0, 0.0)])  # the share is free again
    assert sg.pool_usage()[0] - used0 >= 4 * side * side
    again.close()


@pytest.mark.parametrize("path", ["plain", "bf16x6"])
def test_a_server_gives_its_launch_memory_back(path):
    _reserved()
    used0 = sg.pool_usage()[0]
    srv = sg.Server(1 << 28, slots=2, max_batch=4, path=path)
    for seed in range(6):
        srv.submit(256, 512, 512, seed=seed)
    srv.drain()
    assert sg.pool_usage()[0] > used0
    srv.close()
    _reserved()
    assert sg.pool_usage()[0] == used0


@pytest.mark.parametrize("path", ["plain", "bf16x6", "tf32x3"])
def test_a_server_holds_what_its_header_says_beside_the_budget(path):
    """A small budget and several slots: operands that a plain batch prepares within an
    eighth of the budget, the slab sums of a split batch per slot, and tables."""
    import torch

    _reserved()
    used0 = sg.pool_usage()[0]
    budget, slots = 64 << 20, 3
    srv = sg.Server(budget, slots=slots, max_batch=4, path=path)
    for seed in range(24):
        srv.submit(96 + seed, 768, 4096, seed=seed)
    srv.drain()
    held = sg.pool_usage()[0] - used0
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    share = budget // 8 if path == "plain" else slots * sms * (64 << 10)
    assert held <= share + slots * (4 << 20)
    srv.close()
