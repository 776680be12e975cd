"""Calls of the host path that fail half way, and calls it refuses."""
import pytest
import torch

import llsa_b200
from llsa_b200 import ops, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(N, H=2):
    q, k, v, do = [t.to(DEV) for t in synth.gaussian_qkv(N, 1, H, N, 64, dtype=torch.bfloat16)]
    o, saved = ops._layer(q, k, v, None, None, None, 0.0, 8, 8, 16, 2)
    bwd = lambda d_o, q=q, k=k, v=v, o=o, saved=saved: torch.ops.llsa_b200.layer_bwd(d_o, q, k, v, o, saved, None, None, None, None, None, 0.0, 8, 8, 16, 2,
                                                                                  False)
    return q, k, v, do, o, saved, bwd


def test_a_backward_that_fails_behind_the_fork_joins_the_side_stream():
    """A gradient of the wrong length is found when the index transpose is already on the side stream.  Were the streams not joined on the
    way out, the capture around the call could not end."""
    q, k, v, do, o, saved, bwd = _layer(16384)
    want = bwd(do)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(RuntimeError, match="d_o"):
            bwd(do[:, :, 256:])
        got = bwd(do)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0])
    with pytest.raises(RuntimeError, match="d_o"):
        bwd(do[:, :, 256:])
    assert torch.equal(bwd(do)[0], want[0])


@pytest.mark.parametrize("which", ["q", "k", "v", "o", "saved"])
def test_backward_refuses_a_host_operand(which):
    """What a saved-tensor hook that forgets to bring a tensor back would hand over."""
    q, k, v, do, o, saved, bwd = _layer(4096)
    x = dict(q=q, k=k, v=v, o=o, saved=saved)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        bwd(do, **{which: x[which].cpu()})


def test_operators_refuse_a_host_weight_index_or_table():
    q, k, v, do, o, saved, bwd = _layer(4096)
    w, table = torch.ones(64, device=DEV), torch.ones(4096, 64, device=DEV, dtype=q.dtype)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        llsa_b200.llsa_l2_rms_rope(q, k, v, w.cpu(), w, table)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        llsa_b200.llsa_l2_rms_rope(q, k, v, w, w, table.cpu())
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ops.rms_norm(q, w.cpu())
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ops.rms_rope_pool_pyramid([q, k, v], [w, w.cpu(), None], 1e-5, table, [True, True, False], 16, 2)
    dbg = llsa_b200.llsa_l1_debug(q, k, v, 8, 16)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ops.sparse_indices_attn_res_fwd(q, k, v, dbg["pk"].cpu(), dbg["pv"], dbg["indices"], 8, 16)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ops.sparse_indices_attn_res_scatter_bwd_v2(do, q, k, v, dbg["pk"], dbg["pv"], dbg["o"], dbg["lse"], dbg["indices"].cpu(), 8, 16, 16)


def test_core_backward_refuses_lists_of_another_length():
    q, k, v, do, o, saved, bwd = _layer(4096)
    one = llsa_b200.llsa_l1_debug(q, k, v, 8, 16)
    two = llsa_b200.llsa_l2_debug(q, k, v, 8, 8, 16)
    with pytest.raises(RuntimeError, match="indices"):
        ops.sparse_indices_attn_res_scatter_bwd_v2(do, q, k, v, one["pk"], one["pv"], one["o"], one["lse"], one["indices"], 4, 16, 16)
    with pytest.raises(RuntimeError, match="indices"):
        ops.sparse_indices_attn_res_scatter_2_2_bwd_v2(do, q, k, v, *[two[n] for n in ("pk", "pv", "pk2", "pv2", "o", "lse", "indices", "p_indices")],
                                                       4, 8, 16, 16, 256)
    with pytest.raises(RuntimeError, match="p_indices"):
        ops.sparse_indices_attn_res_scatter_2_2_bwd_v2(do, q, k, v, *[two[n] for n in ("pk", "pv", "pk2", "pv2", "o", "lse", "indices", "p_indices")],
                                                       8, 4, 16, 16, 256)
