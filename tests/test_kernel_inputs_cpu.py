"""What the host hands to kernels that read 16 bytes at a time, checked on the CPU: base addresses and row pitches."""

from types import SimpleNamespace

import pytest
import torch


def _views(n, *shape):
    """bf16 tensors of one shape: aligned, contiguous 4 elements into their storage, transposed, with an odd row pitch, expanded."""
    numel = torch.Size(shape).numel()
    base = torch.arange(numel + 64, dtype=torch.float32).bfloat16()
    yield base[:numel].view(shape)
    yield base[4:4 + numel].view(shape)
    yield base[:numel].view(*shape[:-2], shape[-1], shape[-2]).transpose(-1, -2)
    yield torch.zeros(*shape[:-1], shape[-1] + n).bfloat16()[..., :shape[-1]]
    yield base[1:1 + shape[-1]].expand(shape)


def _readable(t):
    return t.stride(-1) == 1 and t.data_ptr() % 16 == 0 and all(s % 8 == 0 for s, n in zip(t.stride()[:-1], t.shape) if n > 1)


@pytest.mark.parametrize("shape", [(1, 1, 1, 128), (2, 3, 2, 128), (1, 65, 4, 128)])
def test_delta_rule_inputs_are_readable_in_16_byte_pieces(shape):
    from pithtrain_b200.ops.gated_delta_rule import _rows_of_8

    for t in _views(4, *shape):
        got = _rows_of_8(t)
        assert torch.equal(got, t) and _readable(got)
    wide = torch.zeros(*shape[:2], 3 * shape[2] * 128).bfloat16()[..., 128 * shape[2]:256 * shape[2]].unflatten(-1, shape[2:])
    assert _rows_of_8(wide).data_ptr() == wide.data_ptr()  # a slice of a projection is read in place


@pytest.mark.parametrize("n", [1, 5])
def test_mla_inputs_are_readable_in_16_byte_pieces(n):
    from pithtrain_b200.ops import mla

    for t in _views(4, n, 64):
        got = mla._rows(t)
        assert torch.equal(got, t) and _readable(got)
    wide = torch.zeros(n, 200).bfloat16()[:, 72:136]
    assert mla._rows(wide).data_ptr() == wide.data_ptr()
    # one token: the blocks of a projection of odd width are contiguous where they lie
    for block in mla.split_columns(torch.zeros(1, 128 + 20 + 64).bfloat16(), (128, 20, 64)):
        assert mla._rows(block).data_ptr() % 16 == 0


@pytest.mark.parametrize("shape", [(1, 1, 2, 128), (1, 1, 1, 64), (2, 5, 3, 64), (1, 63, 1, 256)])
def test_output_gradients_of_attention_are_readable_in_16_byte_pieces(shape):
    from pithtrain_b200.ops import attention_native as N

    for t in _views(4, *shape):
        got = N._aligned_gradient(t)
        assert torch.equal(got, t) and N._token_major(got)


def test_current_device_predicate(monkeypatch):
    from pithtrain_b200 import _native

    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 1, raising=False)
    on = [SimpleNamespace(is_cuda=True, get_device=lambda d=d: d) for d in (0, 1)]
    assert [_native.on_current_device(t) for t in on] == [False, True]
    assert not _native.on_current_device(torch.zeros(1))


def _fake(*shape, dtype=torch.bfloat16):
    """A tensor that says it is on a CUDA device and has no memory."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    with FakeTensorMode():
        return torch.empty((*shape[:-1], shape[-1] or 8), device="cuda", dtype=dtype)[..., : shape[-1]]  # no elements: of rows that have some


def _host():
    from pithtrain_b200 import _native

    if not _native._HOST_PATH.exists():
        pytest.skip("the host library is not built")
    return _native.host()


def test_host_operators_refuse_operands_elsewhere():
    """A weight, table or index on the host beside activations on the device is refused before anything reads it."""
    h, cpu = _host(), lambda *s: torch.zeros(s, dtype=torch.bfloat16)  # noqa: E731
    x, ids = _fake(8, 64), torch.zeros(8, 2, dtype=torch.int32)
    w1, w2 = _fake(4, 128, 64), _fake(4, 64, 64)
    calls = [
        lambda: h.linear(x, cpu(64, 64), None, None, None),
        lambda: h.linear(x, _fake(64, 64), cpu(64), None, None),
        lambda: h.rmsnorm(x, cpu(64), 1e-6, None, False),
        lambda: h.rmsnorm(x, _fake(64), 1e-6, cpu(8, 64), False),
        lambda: h.qk_norm_rope(_fake(8, 192), cpu(64), cpu(64), _fake(8, 64), _fake(8, 64), None, 1, 1, 64, 1e-6, 8, False),
        lambda: h.qk_norm_rope(_fake(8, 192), None, None, cpu(8, 64), cpu(8, 64), None, 1, 1, 64, 1e-6, 8, False),
        lambda: h.qk_norm_rope(_fake(8, 192), None, None, _fake(8, 64), _fake(8, 64), torch.zeros(8, dtype=torch.int32), 1, 1, 64, 1e-6, 8, False),
        lambda: h.attention(_fake(1, 8, 1, 64), cpu(1, 8, 1, 64), _fake(1, 8, 1, 64), None, None, 1.0, True, 0, 8),
        lambda: h.attention(_fake(1, 8, 1, 64), _fake(1, 8, 1, 64), _fake(1, 8, 1, 64), None, torch.zeros(8, dtype=torch.int32), 1.0, True, 0, 8),
        lambda: h.router(x, ids, 2, 0, True, 1.0),
        lambda: h.moe_experts(x, _fake(8, 2), _fake(8, 2, dtype=torch.int32), w1.new_zeros(w1.shape, device="cpu"), w2, 16, 96, False, 1.0, 0.0, None),
        lambda: h.moe_experts(x, _fake(8, 2), _fake(8, 2, dtype=torch.int32), w1, w2.new_zeros(w2.shape, device="cpu"), 16, 96, False, 1.0, 0.0, None),
        lambda: h.wgrad_into(_fake(8, 64), _fake(8, 64), torch.zeros(64, 64), False),
    ]
    for call in calls:
        with pytest.raises(RuntimeError, match="operands on cuda"):
            call()
    with pytest.raises(RuntimeError, match="must be on a CUDA device"):
        h.linear(cpu(8, 64), cpu(64, 64), None, None, None)


def test_host_operators_refuse_operands_without_memory():
    h, x = _host(), _fake(8, 64)
    for call in (lambda: h.linear(x, _fake(64, 64), None, None, None), lambda: h.rmsnorm(x, _fake(64), 1e-6, None, False), lambda: h.router_picks(x, 2),
                 lambda: h.wgrad_into(x, x, _fake(64, 64, dtype=torch.float32), False)):
        with pytest.raises(RuntimeError, match="no memory"):
            call()


def test_host_operators_refuse_widths_of_zero():
    """Rows of no elements have no number; dividing by their width ended the process."""
    h = _host()
    for x in (_fake(8, 0), _fake(0, 0)):
        with pytest.raises(RuntimeError, match="linear"):
            h.linear(x, _fake(64, 0), None, None, None)
        with pytest.raises(RuntimeError, match="no elements"):
            h.rmsnorm(x, _fake(0), 1e-6, None, False)


def test_shared_memory_is_asked_for_on_each_device(tmp_path):
    """A kernel of one translation unit on three devices, against a runtime that only counts; a refusal is passed on and tried again."""
    import shutil
    import subprocess
    from pathlib import Path

    import pithtrain_b200

    if shutil.which("g++") is None or not Path("/usr/local/cuda/include/cuda_runtime.h").exists():
        pytest.skip("no compiler or no CUDA headers")
    csrc = Path(pithtrain_b200.__file__).parent / "csrc"
    assert not any("static bool" in line and "false" in line for f in csrc.glob("*.cu") for line in f.read_text().splitlines())
    (tmp_path / "t.cpp").write_text("""
#include "host_common.h"
static int device = 0, asked = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++asked; return answer; }
void kernel(int) {}
int main() {
  static pt::SmemLimit limit;
  for (int round = 0; round < 2; ++round)
    for (device = 0; device < 3; ++device)
      if (limit.set(kernel, 1 << 16) != cudaSuccess) return 1;
  if (asked != 3) return 2;
  static pt::SmemLimit other;
  answer = cudaErrorInvalidValue;
  if (other.set(kernel, 1 << 16) != cudaErrorInvalidValue) return 3;
  answer = cudaSuccess;
  return other.set(kernel, 1 << 16) == cudaSuccess && asked == 5 ? 0 : 4;
}
""")
    subprocess.run(["g++", "-std=c++17", f"-I{csrc}", "-I/usr/local/cuda/include", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0
