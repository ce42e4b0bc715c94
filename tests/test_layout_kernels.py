"""The list fill and the fused eps / 1/eps pack of the layout kernels, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("lens", [[], [0], [1], [3, 0, 4, 5], [8191, 8192, 8193],
                                  [17] * 128, [2 + k % 7 for k in range(300)], [5_000_001, 1]])
def test_zero_list(lens):
    """Buffers of every alignment and remainder, empty ones, more than one launch takes:
    exactly their elements become zero."""
    from meep_torch_b200 import _lib as L
    pad = 3
    arena = torch.ones(sum(lens) + pad * (len(lens) + 1), device="cuda")
    want, bufs, o = arena.clone(), [], pad
    for n in lens:
        bufs.append(arena[o:o + n])
        want[o:o + n] = 0
        o += n + pad
    L.zero(L.load(), bufs, _stream())
    assert torch.equal(arena, want)


@pytest.mark.parametrize("nx, ny, pitch", [(1, 1, 4), (7, 13, 16), (33, 128, 128), (901, 1030, 1032)])
def test_pack_eps(nx, ny, pitch):
    from meep_torch_b200 import _lib as L
    lib = L.load()
    g = torch.Generator().manual_seed(nx)
    src = (1 + 11 * torch.rand((nx, ny), generator=g)).cuda()
    src[0, 0] = 1e-40                                  # a denormal: 1/eps overflows to inf
    eps, inv = (torch.full((nx, pitch), 7.0, device="cuda") for _ in range(2))
    L.check(lib.mtb_pack_eps(L.ptr(src), nx, ny, pitch, L.ptr(eps), L.ptr(inv), _stream()), "pack")
    for box, ref in ((eps, src), (inv, torch.reciprocal(src))):
        assert torch.equal(box[:, :ny], ref) and not box[:, ny:].any()
