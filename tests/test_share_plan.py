"""How stage 1 deals the groups of a batch to its CTAs and where stage 2 looks for the results: the plan of the library
(host twin of what both kernels compute) held to what the kernels assume of it, over random lengths and split counts."""
import ctypes as C
import random

import pytest

from open_ommx_serve_b200 import _lib

SMS = 148


def plan(groups, splits, bound):
    """``bound``: the call's max_seq_len in multiples of the longest sequence."""
    lens = (C.c_int32 * len(groups))(*[32 * g for g in groups])
    ctas, per = C.c_int32(), C.c_int32()
    limit = _lib.load().ommx_b200_host_share_plan(lens, len(groups), splits, 32 * max(groups) * bound, SMS, C.byref(ctas), C.byref(per))
    assert limit == 128
    return limit, ctas.value, per.value


def pieces_of(groups, splits, ctas, per):
    """(cta, sequence, slot, first group, groups) of every piece, as stage 1 lists them."""
    out = []
    if per == 0:                                            # split x % S of sequence x / S, dealt out one by one
        for x in range(len(groups) * splits):
            b, s = divmod(x, splits)
            size = -(-groups[b] // splits)
            if s * size < groups[b]:
                out.append((x % ctas, b, s, s * size, min(size, groups[b] - s * size)))
        return out
    at = 0
    for b, n in enumerate(groups):
        for cta in range(at // per, (at + n - 1) // per + 1 if n else at // per):
            lo, hi = max(at, cta * per), min(at + n, (cta + 1) * per)
            out.append((cta, b, cta - at // per, lo - at, hi - lo))
        at += n
    return out


def check(groups, splits, bound=1):
    limit, ctas, per = plan(groups, splits, bound)
    pieces = pieces_of(groups, splits, ctas, per)
    count, slots, covered, before = {}, {}, [0] * len(groups), 0
    for cta, b, slot, first, n in pieces:
        assert 0 <= cta < ctas and n > 0 and first == covered[b]           # every group once, in order
        covered[b] += n
        count[cta] = count.get(cta, 0) + 1
        slots.setdefault(b, []).append(slot)
    assert covered == list(groups)
    assert max(count.values(), default=0) <= limit, (max(count.values()), per, ctas)
    for b, n in enumerate(groups):                          # stage 2 reads slots 0 .. count - 1 of the caller's S
        if n == 0:
            want = 0
        elif per == 0:
            want = -(-n // -(-n // splits))
        else:
            want = (before + n - 1) // per - before // per + 1
        assert slots.get(b, []) == list(range(want)) and want <= splits
        before += n


@pytest.mark.parametrize("long", [129, 130, 200, 254, 300])
@pytest.mark.parametrize("n", [200, 220, 300, 1000])
@pytest.mark.parametrize("at", [0, 100, -1])
def test_many_short_sequences_beside_a_longer_one(n, long, at):
    """The share that the longest sequence asks for holds more short sequences than a CTA can list."""
    groups = [1] * n
    groups[at] = long
    for splits in (2, 3, 5):
        check(groups, splits)
        check(groups, splits, 16)


def test_a_share_of_as_many_sequences_as_a_cta_lists_is_kept():
    groups = [1] * 299 + [129]
    limit, ctas, per = plan(groups, 2, 1)
    pieces = pieces_of(groups, 2, ctas, per)
    assert per == limit and sum(1 for p in pieces if p[0] == 0) == limit


@pytest.mark.parametrize("seed", range(300))
def test_every_group_is_dealt_once_and_found_again(seed):
    rng = random.Random(seed)
    batch = int(round(600 ** rng.random())) if rng.random() < 0.7 else rng.randint(129, 600)
    hi = int(round(512 ** rng.random()))
    kind = rng.randrange(3)
    groups = [rng.randint(0 if kind else hi, hi) for _ in range(batch)]
    if kind == 2:
        groups = [rng.randint(0, 2) for _ in range(batch)]
        groups[rng.randrange(batch)] = hi
    if max(groups) == 0:
        groups[0] = 1
    auto = _lib.load().ommx_b200_auto_num_kv_splits(32 * max(groups), batch, 8)
    for splits in {auto, 1, rng.randint(2, 8), int(round(1024 ** rng.random()))}:
        check(groups, splits, rng.choice((1, 1, 2, 16)))


def launch(groups, splits, clusters=None, sms=SMS):
    lens = (C.c_int32 * len(groups))(*[32 * g for g in groups])
    out = _lib.LaunchPlan()
    at_once = (C.c_int32 * 3)(*clusters) if clusters else None
    rc = _lib.load().ommx_b200_host_launch_plan(lens, len(groups), splits, 32 * max(groups), sms, at_once, C.byref(out))
    assert rc == 128, _lib.last_error()
    return out


@pytest.mark.parametrize("clusters", [None, (74, 33, 15), (74, 32, 0), (70, 0, 0), (0, 0, 0), (5, 3, 1)])
@pytest.mark.parametrize("groups,splits", [([128], 8), ([512], 32), ([64, 20, 33, 40] * 2, 4), ([256, 130, 200, 180], 16), ([64] + [1] * 60, 2),
                                           ([2048], 147), ([1024] * 8, 18)])
def test_launch_and_shares_agree(groups, splits, clusters):
    """The clusters of a launch run at once, a share is one CTA's or one whole cluster's, and every share has its CTAs."""
    p = launch(groups, splits, clusters)
    assert p.ctas % p.cluster == 0 and p.ctas_per_share in (1, p.cluster) and p.shares * p.ctas_per_share == p.ctas <= SMS
    if p.cluster > 1:
        assert p.ctas // p.cluster <= (clusters or (74, 33, 15))[p.cluster // 4]
    if not clusters:
        assert plan(groups, splits, 1)[1:] == (p.shares, p.groups_per_share)


def test_few_slots_take_clusters_where_there_are_any():
    assert launch([128], 8).cluster > 1 and launch([128], 8).ctas_per_share > 1
    assert launch([2048], 147).cluster == 1
    alone = launch([128], 8, (0, 0, 0))
    assert (alone.ctas, alone.cluster, alone.shares, alone.ctas_per_share) == (128, 1, 128, 1)


def test_launch_plan_refuses_more_clusters_than_sms():
    lens = (C.c_int32 * 1)(32)
    for bad in ((75, 0, 0), (0, 38, 0), (0, 0, 19), (-1, 0, 0)):
        assert _lib.load().ommx_b200_host_launch_plan(lens, 1, 1, 32, SMS, (C.c_int32 * 3)(*bad), C.byref(_lib.LaunchPlan())) == -1


@pytest.mark.gpu
def test_launches_count_on_the_clusters_that_this_device_runs():
    """Against the driver's answer for a kernel of ours that takes a whole SM."""
    import torch
    from cuda.bindings import driver, nvrtc

    def ok(result):
        assert int(result[0]) == 0, result
        return result[1:] if len(result) > 2 else (result[1] if len(result) > 1 else None)

    torch.zeros(1, device="cuda")
    prog = ok(nvrtc.nvrtcCreateProgram(b'extern "C" __global__ void alone(float *p) { extern __shared__ float s[]; if (p) p[0] = s[0]; }',
                                       b"alone.cu", 0, [], []))
    ok(nvrtc.nvrtcCompileProgram(prog, 1, [b"--gpu-architecture=sm_100a"]))
    image = b" " * ok(nvrtc.nvrtcGetCUBINSize(prog))
    ok(nvrtc.nvrtcGetCUBIN(prog, image))
    fn = ok(driver.cuModuleGetFunction(ok(driver.cuModuleLoadData(image)), b"alone"))
    smem = 200 * 1024
    ok(driver.cuFuncSetAttribute(fn, driver.CUfunction_attribute.CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, smem))
    at_once = []
    for size in (2, 4, 8):
        attr = driver.CUlaunchAttribute()
        attr.id = driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION
        attr.value.clusterDim.x, attr.value.clusterDim.y, attr.value.clusterDim.z = size, 1, 1
        cfg = driver.CUlaunchConfig()
        cfg.gridDimX, cfg.gridDimY, cfg.gridDimZ = size, 1, 1
        cfg.blockDimX, cfg.blockDimY, cfg.blockDimZ = 768, 1, 1
        cfg.sharedMemBytes, cfg.attrs, cfg.numAttrs = smem, [attr], 1
        at_once.append(ok(driver.cuOccupancyMaxActiveClusters(fn, cfg)))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = set()
    for groups, splits in (([2048], 8), ([512], 32), ([64] + [1] * 60, 2), ([512], 72), ([2048], 147)):
        here, want = launch(groups, splits, sms=0), launch(groups, splits, at_once, sms)
        assert all(getattr(here, f) == getattr(want, f) for f, _ in _lib.LaunchPlan._fields_)
        if here.cluster > 1 and here.ctas // here.cluster == at_once[here.cluster // 4]:
            sizes.add(here.cluster)
    assert sizes == {2, 4, 8}
