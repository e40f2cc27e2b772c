"""Decode steps of the Reasoner on the kernels: what surrounds the layers (csrc/step_edges.cu) and the order of the launches."""
import pytest
import torch

from cosmos_b200 import ops
from cosmos_b200.config import get_model_config
from cosmos_b200.serve.decoder import TPDecoder

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(autouse=True)
def _status_clean():
    ops.load_extension()
    yield
    torch.cuda.synchronize()
    ops.check_status()


def _decoder(batch, prompt=40, room=16, **kw):
    cfg = get_model_config("tiny128", **{"n_layers": 2, **kw})
    dec = TPDecoder(cfg, 1, 0, None, DEV, page_size=16, max_batch=batch, max_len=prompt + room)
    dec.prefill_synthetic(batch, prompt, room)
    return dec


@pytest.mark.parametrize("batch,d,inner", [(1, 512, 8192), (3, 1024, 16384), (33, 512, 16384), (128, 2048, 8192)])
def test_eager_step_behind_a_kernel_that_writes_a_weight(batch, d, inner):
    """The GEMM in front of an eager step writes the weight that the step's first projection reads (and reads ahead), with
    nothing between them; again with that weight long in place. The same bits: the same kernels on the same numbers."""
    dec = _decoder(batch, d_model=d, n_heads=d // 128, n_kv_heads=2, ffn_dim=2 * d)
    tokens, lens = dec.tokens.clone(), dec.lens.clone()
    w = dec.layers[0]["wqkv"]
    right = (torch.randn(d, inner, device=DEV) * inner ** -0.5).bfloat16()
    dec.step()
    for seed in range(3):
        torch.manual_seed(seed)
        left = (torch.randn(w.shape[0], inner, device=DEV) * 0.05).bfloat16()
        dec.tokens.copy_(tokens)
        dec.lens.copy_(lens)
        ops.gemm(left, right, out=w)
        dec.step()
        got = dec.last_logits.clone()
        torch.cuda.synchronize()
        dec.tokens.copy_(tokens)
        dec.lens.copy_(lens)
        torch.cuda.synchronize()
        dec.step()
        assert torch.equal(got, dec.last_logits)
