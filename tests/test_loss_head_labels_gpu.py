"""Labels outside [0, classes) in the loss head: the fused call against softmax,
cross entropy and its gradient as separate calls, bit for bit (such a sample's
loss is NaN and nothing is subtracted from its gradient).  A row is held by
threads x vectors slots, more than it has classes: a label that is the number
of an unused slot is as wrong as any other."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (threads per row, 16-byte vectors per thread), the smallest that holds the row is taken
HOLDERS = [(32, 1), (32, 2), (32, 4), (128, 2), (128, 4), (256, 4), (512, 4), (1024, 4), (1024, 8)]


def slots(classes):
    vectors = (classes + 3) // 4
    return next((4 * t * v for t, v in HOLDERS if vectors <= t * v), classes)


@pytest.mark.parametrize("classes", [1, 10, 12, 127, 128, 129, 300, 1000, 1001, 5002, 20004, 32767, 32770])
@pytest.mark.parametrize("offset", [0, 1])
def test_labels_out_of_range(classes, offset):
    from singa_b200 import _lib
    held = slots(classes)
    labels = [0, -1, classes, classes + 1, (classes + held) // 2, held - 1, held, held + 1, 2 ** 31 - 1, -2 ** 31,
              classes - 1]
    batch = len(labels)
    gen = torch.Generator(device="cuda").manual_seed(classes)
    x = torch.randn(batch * classes + offset, device="cuda", generator=gen)[offset:]
    t = torch.tensor(labels, dtype=torch.int32, device="cuda")
    p1, p2, g1, g2 = [torch.full((batch * classes + offset,), 7.0, device="cuda")[offset:] for _ in range(4)]
    l1, l2 = torch.full((batch,), 7.0, device="cuda"), torch.full((batch,), 7.0, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    scale = 1.0 / batch

    def call(name, *args):
        _lib.call(name, *[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args], stream)

    call("sgb_softmax_rows_f32", x, p1, batch, classes)
    call("sgb_cross_entropy_f32", 1, batch, classes, p1, t, l1)
    call("sgb_softmax_cross_entropy_grad_f32", 1, batch, classes, p1, t, scale, g1)
    call("sgb_softmax_cross_entropy_fused_f32", x, t, batch, classes, scale, p2, l2, g2)
    for got, want in ((p2, p1), (l2, l1), (g2, g1)):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    known = torch.tensor([0 <= label < classes for label in labels], device="cuda")
    assert torch.equal(torch.isnan(l2), ~known)
