"""Tensors that a kernel would read or write outside what is there - in plain host memory, or too few - are refused before
anything is launched."""
import pytest
import torch

from helpers import Case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    return Case([300], seed=4)


@pytest.mark.parametrize("name", ["k_base", "k_scale", "k_zp", "k_obmp", "k_oval", "k_fp4_mapscale", "k_fp4_mapcenter", "v_main", "v_scale", "v_zp"])
def test_decode_refuses_a_plane_on_the_host(case, name, monkeypatch):
    monkeypatch.setitem(case.planes, name, case.planes[name].cpu())
    with pytest.raises(ValueError, match=name):
        case.run()


def test_decode_refuses_a_status_word_on_the_host(case):
    with pytest.raises(ValueError, match="status"):
        case.run(status=torch.zeros(1, dtype=torch.int32))
    pinned = torch.zeros(1, dtype=torch.int32).pin_memory()                 # which the GPU can reach
    case.run(status=pinned)
    assert int(pinned) == 0


def test_pack_refuses_values_planes_and_status_on_the_host():
    from open_ommx_serve_b200.attention.pack import alloc_planes, ommx_pack_kv_into
    K = torch.randn(64, 2, 128, device="cuda").bfloat16()
    planes = alloc_planes(4, 2, 2, 128)
    kw = dict(outliers_per_vector=6)
    with pytest.raises(ValueError, match="V is on cpu"):
        ommx_pack_kv_into(K, K.cpu(), planes, **kw)
    with pytest.raises(ValueError, match="status"):
        ommx_pack_kv_into(K, K, planes, status=torch.zeros(1, dtype=torch.int32), **kw)
    for name in [n for n, t in planes.items() if t is not None]:
        with pytest.raises(ValueError, match=name):
            ommx_pack_kv_into(K, K, {**planes, name: planes[name].cpu()}, **kw)
    ommx_pack_kv_into(K, K, planes, **kw)


@pytest.mark.parametrize("which", range(4))
def test_gather_refuses_indices_and_buffers_on_the_host(which):
    from open_ommx_serve_b200.attention.kv_pool import MultiSeqKVPool
    pool = MultiSeqKVPool(128, 2, 2, 256)
    args = [torch.zeros(2, dtype=torch.int64), torch.zeros(2, 8, dtype=torch.int64), torch.zeros(2, 8, 2, 128, dtype=torch.bfloat16),
            torch.zeros(2, 8, 2, 128, dtype=torch.bfloat16)]
    args = [t if i == which else t.cuda() for i, t in enumerate(args)]
    with pytest.raises(ValueError, match="CUDA"):
        pool._gather_tail(*args)


def test_gather_refuses_a_selection_that_is_too_short():
    """One entry of ``sel`` is read for every row of tail indices."""
    from open_ommx_serve_b200.attention.kv_pool import MultiSeqKVPool
    pool = MultiSeqKVPool(128, 2, 4, 256)
    buf = torch.zeros(2, 8, 2, 128, dtype=torch.bfloat16, device="cuda")
    lens = torch.zeros(2, dtype=torch.int32, device="cuda")
    tidx = torch.zeros(2, 8, dtype=torch.int64, device="cuda")
    with pytest.raises(ValueError, match="1 slots for 2 rows"):
        pool.decode_inputs_captured(torch.arange(1, device="cuda"), lens, lens, tidx, buf, buf.clone(), 0)
    for n in (2, 3):                                       # a longer one's first entries count
        pool.decode_inputs_captured(torch.arange(n, device="cuda"), lens, lens, tidx, buf, buf.clone(), 0)


def test_merge_refuses_lse_on_the_host():
    from open_ommx_serve_b200 import merge_attention_states
    with pytest.raises(ValueError, match="lse_parts"):
        merge_attention_states(torch.zeros(2, 4, 128, device="cuda"), torch.zeros(2, 4))
