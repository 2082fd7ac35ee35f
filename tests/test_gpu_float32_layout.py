"""One-call encoder at lengths whose convolution runs in float32: either layout in the workspace that is asked for it."""
import pytest
import torch

from m2_b200 import _lib, ops
from m2_b200.encoder import M2BertConfig, M2BertModel
from tests.test_gpu_determinism import DEV, guarded, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L", [(6, 1531), (40, 301), (3, 129)])
def test_encoder_in_both_layouts(B, L):
    D, I = 256, 512
    torch.manual_seed(L)
    model = M2BertModel(M2BertConfig(vocab_size=96, hidden_size=D, intermediate_size=I, num_hidden_layers=2, max_position_embeddings=2048,
                                     long_conv_l_max=2048, hyena_filter_order=16)).eval().to(DEV)
    ids = torch.randint(0, 96, (B, L), device=DEV)
    out = {}
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        plan = model._make_plan(B, L, torch.device(DEV))
        assert plan.args.kind == 0 and plan.args.padded == ops.longconv_padded(B, L, D)
        for padded in (0, 1):
            for size in (_lib.lib().m2_encoder_workspace_kind(0, padded, B, L, D, I), _lib.lib().m2_encoder_workspace(B, (L + 7) // 8 * 8, D, I)):
                work, check = guarded((size // 4 + 64,), torch.float32)
                start = (work.data_ptr() + 255) // 256 * 256
                work.view(torch.int32)[(start - work.data_ptr() + size) // 4:] = 0x5A5A5A5A
                y = torch.empty((B, L, D), device=DEV)
                a = _lib.EncoderArgs.from_buffer_copy(plan.args)
                a.padded, a.workspace, a.out, a.embed.input_ids = padded, start, y.data_ptr(), ids.data_ptr()
                native(_lib.lib().m2_encoder_fwd, a)
                torch.cuda.synchronize()
                check()
                assert (work.view(torch.int32)[(start - work.data_ptr() + size) // 4:] == 0x5A5A5A5A).all()
                assert torch.equal(out.setdefault(padded, y), y)
        assert torch.equal(out[plan.args.padded], model(ids)[0])
    # two layers of bf16 roundings, a few in a thousand of which fall the other way
    assert ((out[0] - out[1]).norm() / out[0].norm()).item() < 5e-3
    assert ops.device_status() == 0
