"""The native binding of the Python caller: what it raises, what it accepts, how it uses a workspace. Tensors of these tests are
on the CPU, so a call ends at the latest before its second phase."""
import pytest
import torch


def test_torch_errors_keep_their_type_and_message(ops):
    """An allocation that torch refuses is reported as torch reports it, without a C++ stack trace."""
    x = torch.zeros(1, 1, 4, 4)
    for size in ((2 ** 31 - 1, 2 ** 31 - 1), (-3, 5)):
        with pytest.raises(RuntimeError) as plain:
            torch.empty((2 ** 20, 2 ** 20) + size if size[0] > 0 else (1, 1) + size)
        with pytest.raises(RuntimeError) as bound:
            ops.upsample_bilinear2d(x.expand(2 ** 20, 2 ** 20, 4, 4) if size[0] > 0 else x, size)
        assert type(bound.value) is type(plain.value)
        assert str(bound.value).splitlines()[0][:30] == str(plain.value).splitlines()[0][:30]
        assert "Exception raised from" not in str(bound.value)


@pytest.mark.gpu
def test_out_of_memory_is_torchs(ops, dev):
    x = torch.zeros(1, 1, 4, 4, device=dev)
    with pytest.raises(torch.OutOfMemoryError):
        ops.upsample_nearest2d(x, (2 ** 21, 2 ** 21))
    assert ops.upsample_nearest2d(x, (8, 8)).shape == (1, 1, 8, 8)  # and the device works on
