"""Lengths whose convolution runs in float32: one kernel for all batches, so that a sequence's result does not depend on what it is
batched with, and the whole encoder inside the workspace that is asked for it."""
import pytest
import torch

from m2_b200 import _lib, ops
from m2_b200.encoder import M2BertConfig, M2BertModel
from tests.test_gpu_determinism import DEV, guarded, native
from tests.test_gpu_precision import mixer

pytestmark = pytest.mark.gpu


def bf16(f, *args):
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        return f(*args)[0]


@pytest.mark.parametrize("L,batches", [(131, (1, 4, 12, 16, 24, 32)), (301, (1, 8, 40)), (1531, (1, 6)), (2047, (1, 10))])
def test_results_do_not_depend_on_the_batch(L, batches):
    m, _, u = mixer(L, 256, max(batches))
    alone = bf16(m, u[:1])
    assert ops.longconv_pick(1, L, torch.bfloat16, 256) == 0
    for B in batches:
        assert torch.equal(bf16(m, u[:B])[:1], alone)


@pytest.mark.parametrize("B,L", [(6, 1531), (40, 301), (3, 129)])
def test_encoder_stays_in_its_workspace(B, L):
    D, I = 256, 512
    torch.manual_seed(L)
    model = M2BertModel(M2BertConfig(vocab_size=96, hidden_size=D, intermediate_size=I, num_hidden_layers=2, max_position_embeddings=2048,
                                     long_conv_l_max=2048, hyena_filter_order=16)).eval().to(DEV)
    ids = torch.randint(0, 96, (B, L), device=DEV)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        plan = model._make_plan(B, L, torch.device(DEV))
        size = _lib.lib().m2_encoder_workspace(B, (L + 7) // 8 * 8, D, I)
        work, check = guarded((size // 4 + 64,), torch.float32)
        skip = -work.data_ptr() % 256
        behind = work.view(torch.int32)[(skip + size) // 4:]
        behind.fill_(0x5A5A5A5A)
        y = torch.empty((B, L, D), device=DEV)
        a = _lib.EncoderArgs.from_buffer_copy(plan.args)
        a.workspace, a.out, a.embed.input_ids = work.data_ptr() + skip, y.data_ptr(), ids.data_ptr()
        native(_lib.lib().m2_encoder_fwd, a)
        torch.cuda.synchronize()
        check()
        assert (behind == 0x5A5A5A5A).all() and torch.equal(y, model(ids)[0])
        assert torch.equal(y[:1], model(ids[:1])[0])
    assert ops.device_status() == 0
