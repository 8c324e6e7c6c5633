"""The C entry of the general rotation and cache write without a table of frequencies: every value passes, whatever rotary width is
named (csrc/rope_cache.cu); on the path of eight values a thread and on the general one."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pad", [0, 1])                    # rows that start on 16-byte borders, and rows that do not
@pytest.mark.parametrize("interleaved", [0, 1])
def test_values_pass_without_a_table(pad, interleaved):
    from gollmgo_b200.csrc import ops
    T, nh, nkv, d, page = 5, 2, 1, 32, 16
    width = (nh + 2 * nkv) * d
    rows = torch.randn(T, width + pad, device="cuda").bfloat16()
    want = rows.clone()
    k, v = (torch.zeros(1, nkv, page, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    at = torch.arange(T, dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)  # noqa: E731
    rc = ops.lib().gg_rope_kv_write_x(p(rows), ctypes.c_longlong(rows.stride(0)), ops.dtype_code(rows.dtype), p(at), p(at), p(None),
                                      ctypes.c_float(1.0), p(None), p(k), p(v), T, nh, nkv, d, nkv, d, 16, page, interleaved, 1,
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(rows, want)
    assert torch.equal(k[0, 0, :T], want[:, nh * d:(nh + 1) * d]) and torch.equal(v[0, 0, :T], want[:, (nh + 1) * d:(nh + 2) * d])
