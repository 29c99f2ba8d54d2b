"""CPU: how the k-quant kernel for 2 to 15 tokens deals its ring of weights.

Groups of warps walk the ring's positions in turn and wait for a slot by the parity of its lap.  Such a
wait passes at once while the slot is still a whole lap behind, so a ring that wraps is right only if
every slot belongs to one group: the stages are a multiple of the groups.  Checked over the sizes the
entry points take, on the host arithmetic the launch uses (148 SMs, 227 KB of shared memory)."""
import ctypes as C
import random

import pytest

from hesper_b200 import _lib

SMS, SMEM = 148, 232448
Q8_0, Q4_K = 8, 12


class Plan:
    def __init__(self):
        self.f = _lib.load().hb200_kquant_few_tokens_plan
        self.out = [(C.c_int * 4)() for _ in range(4)]

    def __call__(self, fmt, K, Ns, M, gate_up=0):
        n = len(Ns)
        assert self.f(fmt, K, (C.c_int * n)(*Ns), n, gate_up, M, SMS, SMEM, *self.out) == 0, (fmt, K, Ns, M)
        return [tuple(o[s] for o in self.out) for s in range(n)]


def check(plan, what):
    for stages, groups, tiles, total in plan:
        assert 1 <= groups and groups * tiles <= 16 and 1 <= stages <= 32, (what, plan)
        # a ring that never wraps shows every wait a fresh slot
        assert stages >= total or (groups <= stages and stages % groups == 0), (what, plan)


@pytest.mark.parametrize("fmt", [Q4_K, Q8_0])
@pytest.mark.parametrize("M", [2, 15])  # one and two columns of 8 tokens
def test_a_slot_belongs_to_one_group_of_warps(fmt, M):
    plan = Plan()
    for K in (256, 1024, 2560, 4096, 9216, 16384):
        for N in range(1, 14001):
            check(plan(fmt, K, [N], M), (K, N))
            if N % 3 == 0:
                check(plan(fmt, K, [N // 2] * 2, M, 1), (K, N // 2, "gate/up"))
    rng = random.Random(fmt + M)
    for _ in range(30000):
        K = 256 * rng.randint(1, 64)
        Ns = [round(2 ** rng.uniform(0, 13.8)) for _ in range(rng.randint(2, 4))]
        check(plan(fmt, K, Ns, M), (K, Ns))


@pytest.mark.parametrize("fmt,K,Ns,M,gate_up", [
    # rings of fewer stages than warps per tile: a group would start a lap ahead of the others
    (Q8_0, 4096, [2304], 15, 0), (Q8_0, 9216, [2304], 9, 0), (Q8_0, 4096, [1152, 1152], 12, 1),
    (Q8_0, 4096, [1536, 384, 384], 12, 0), (Q4_K, 4096, [11000, 16], 3, 0),
    # rings that wrap several times
    (Q4_K, 10240, [2560], 15, 0), (Q8_0, 10240, [2560], 7, 0),
    # two passes of rows per CTA, wrapping between and inside them
    (Q4_K, 4096, [148 * 128 + 37], 3, 0), (Q8_0, 4096, [148 * 64 + 11] * 2, 12, 1),
])
def test_shapes_of_the_gpu_tests_wrap(fmt, K, Ns, M, gate_up):
    """The GPU tests use these: each has a tensor whose ring wraps."""
    p = Plan()(fmt, K, Ns, M, gate_up)
    check(p, Ns)
    assert any(stages < total for stages, _, _, total in p), p


def test_outside_of_the_kernel():
    f, out = _lib.load().hb200_kquant_few_tokens_plan, [(C.c_int * 4)() for _ in range(4)]
    one = (C.c_int * 1)(100)
    for K, M in ((2560, 1), (2560, 16), (2500, 4), (65792, 4)):
        assert f(Q4_K, K, one, 1, 0, M, SMS, SMEM, *out) == -3
    assert f(99, 2560, one, 1, 0, 4, SMS, SMEM, *out) == -1
    assert f(Q4_K, 2560, (C.c_int * 1)(0), 1, 0, 4, SMS, SMEM, *out) == -1
