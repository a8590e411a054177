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


class _Recorder:
    """A workspace of the caller's own: `get` alone, which may return a tensor, another buffer or nothing."""

    def __init__(self, buf):
        self.buf_of, self.asked = buf, []

    def get(self, nbytes):
        self.asked.append(nbytes)
        return self.buf_of, nbytes


class _Buffer:
    def data_ptr(self):
        return 4096


@pytest.mark.parametrize("buf", [torch.zeros(1 << 16, dtype=torch.uint8), _Buffer(), None])
def test_any_object_with_get_is_a_workspace(ops, buf):
    ws = _Recorder(buf)
    with pytest.raises(ValueError, match="cuda"):  # the call has come as far as the stream
        ops.upsample_bilinear2d(torch.zeros(1, 1, 5, 5), (9, 9), workspace=ws)
    assert len(ws.asked) == 1 and ws.asked[0] > 0


def test_a_workspace_that_overrides_get_is_asked(ops):
    class Counting(ops.Workspace):
        calls = 0

        def get(self, nbytes):
            Counting.calls += 1
            return super().get(nbytes)

    ws = Counting("cpu")
    for _ in range(2):
        with pytest.raises(ValueError, match="cuda"):
            ops.upsample_bilinear2d(torch.zeros(1, 1, 5, 5), (9, 9), workspace=ws)
    assert Counting.calls == 2


def test_a_workspace_grows_and_keeps_its_buffer(ops):
    ws = ops.Workspace("cpu")
    sizes = []
    for extent in (5, 40, 9):
        with pytest.raises(ValueError, match="cuda"):
            ops.upsample_bilinear2d(torch.zeros(1, 1, extent, extent), (2 * extent + 1,) * 2, workspace=ws)
        sizes.append(ws.buf.numel())
    assert sizes[0] < sizes[1] == sizes[2]


def test_a_failing_get_is_reported(ops):
    class Failing:
        def get(self, nbytes):
            raise LookupError("no room")

    with pytest.raises(LookupError, match="no room"):
        ops.upsample_bilinear2d(torch.zeros(1, 1, 5, 5), (9, 9), workspace=Failing())


@pytest.mark.parametrize("mode,pad", [(0.0, 1.0), (True, False), (torch.tensor(0), 2), ("1", "0")])
def test_grid_modes_are_taken_as_int_takes_them(ops, mode, pad):
    x, grid = torch.zeros(1, 1, 4, 4), torch.zeros(1, 3, 3, 2)
    with pytest.raises(ValueError, match="cuda"):
        ops.grid_sampler2d(x, grid, mode, pad)
    with pytest.raises(ValueError, match="cuda"):
        ops.grid_sampler2d_backward(torch.zeros(1, 1, 3, 3), x, grid, mode, pad)


@pytest.mark.parametrize("scales", [(1, 2), ("1.5", 2.0), torch.tensor([1.5, 2.0]), [True, 2.5]])
def test_scales_are_taken_as_float_takes_them(ops, scales):
    with pytest.raises(ValueError, match="cuda"):
        ops.upsample_bilinear2d(torch.zeros(1, 1, 5, 5), (9, 9), scales=scales)


def test_refusals(ops):
    x = torch.zeros(1, 1, 5, 5)
    with pytest.raises(KeyError):
        ops.upsample_nearest2d(x, (9, 9), fmt="NWHC")
    with pytest.raises(KeyError):
        ops.upsample_nearest2d(x.to(torch.complex64), (9, 9))
    with pytest.raises(TypeError):
        ops.upsample_nearest2d([1.0], (9, 9))
    with pytest.raises(TypeError):
        ops.upsample_nearest2d(x, (9.5, 9))
    with pytest.raises(IndexError):
        ops.upsample_nearest2d(x, (9,))
    with pytest.raises(ops.AclnnError) as e:
        ops.upsample_nearest2d(x.to(torch.float64), (9, 9), out=torch.zeros(1, 1, 9, 9, dtype=torch.float64))
    assert e.value.status == 161002 and "GetWorkspaceSize returned 161002" in str(e.value)


@pytest.mark.gpu
def test_out_of_memory_is_torchs(ops, dev):
    x = torch.zeros(1, 1, 4, 4, device=dev)
    with pytest.raises(torch.OutOfMemoryError):
        ops.upsample_nearest2d(x, (2 ** 21, 2 ** 21))
    assert ops.upsample_nearest2d(x, (8, 8)).shape == (1, 1, 8, 8)  # and the device works on
