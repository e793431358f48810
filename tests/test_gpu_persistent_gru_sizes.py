"""The persistent GRU kernels at the edges of their ranges: one and two time steps, batches on both sides of the
16-entry tile and of the three-entry packs, hidden sizes with half K tiles and on both sides of every change of the
number of blocks per group, weights that spill from tensor memory into shared memory. Against `torch.nn.GRU` in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,H,nd", [
    (1, 1, 128, 1), (2, 16, 256, 2), (2, 17, 384, 2), (3, 3, 640, 1), (7, 17, 512, 2), (7, 15, 512, 1), (12, 32, 640, 2),
    (9, 2, 768, 2), (33, 31, 896, 1), (20, 9, 1024, 2), (40, 32, 1024, 2),
])
def test_edges_match_torch_gru(T, B, H, nd):
    from tensorflow_allreduce_b200.ops import persistent_gru as pg

    if not pg.supported(T, B, H, nd):
        pytest.skip("persistent GRU kernels need a compute-capability-10 GPU with enough SMs")
    old = torch.backends.cuda.matmul.allow_tf32, torch.backends.cudnn.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = torch.backends.cudnn.allow_tf32 = False
    try:
        torch.manual_seed(T * 1000 + H + B)
        rnn = torch.nn.GRU(40, H, bidirectional=(nd == 2)).cuda()
        x = torch.randn(T, B, 40, device="cuda", requires_grad=True)
        y_ref, _ = rnn(x)
        y = pg.gru_forward(rnn, x)
        with torch.no_grad():
            assert torch.equal(pg.gru_forward(rnn, x), y)         # without the saved activations
        g = torch.randn_like(y_ref)
        wrt = [x] + list(rnn.parameters())
        ref, got = torch.autograd.grad(y_ref, wrt, g), torch.autograd.grad(y, wrt, g)
        pg.check_status()
        for a, b in zip((y_ref, *ref), (y, *got)):
            assert (a - b).norm().item() <= 2e-3 * (a.norm().item() + 1e-6)
    finally:
        torch.backends.cuda.matmul.allow_tf32, torch.backends.cudnn.allow_tf32 = old
