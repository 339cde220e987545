"""Cache writer against the numpy oracle, byte for byte, where a product stands in for a division: divisors at the ends of the
fp32 range (which take the division), powers of two, and block maxima that put the scale on an E4M3 rounding boundary."""
import numpy as np
import pytest
import torch

import mla_oracle as O
import nvfp4_mla_b200 as mla

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scales", [(1.0, 1.0), (1.0 / 3, 0.1), (2.0 ** -20, 2.0 ** 12), (6.5 / 2688, 6.5 / 448), (1e-33, 1e-33), (1e32, 1e32)])
def test_bytes_equal_oracle(scales):
    ckv_scale, kpe_scale = scales
    g = torch.Generator().manual_seed(3)
    n, ps = 512, 64
    ckv = torch.randn(n, 512, generator=g)
    # block maxima of exactly 6 * ckv_scale * (midpoints between E4M3 values), as far as BF16 holds them
    mid = torch.tensor([(8 + k + 0.5) / 8 * 2.0 ** e for e in range(-6, 8) for k in range(8)])
    blocks = ckv.view(n, 32, 16)
    blocks[:128] *= (mid[torch.randint(0, mid.numel(), (128, 32), generator=g)] / blocks[:128].abs().amax(-1))[..., None] * 6
    ckv = (ckv * ckv_scale).bfloat16()
    kpe = (torch.randn(n, 64, generator=g) * 50 * kpe_scale).bfloat16()
    dev = "cuda"
    caches = (torch.zeros(n // ps, ps, 256, dtype=torch.uint8, device=dev),
              torch.zeros(n // ps, ps, 32, dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn),
              torch.zeros(n // ps, ps, 64, dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn))
    pos = torch.arange(n, dtype=torch.int32, device=dev)
    mla.quantize_append_paged_mla_kv_cache(ckv.to(dev), kpe.to(dev), torch.zeros_like(pos), pos, *caches,
                                           torch.arange(n // ps, dtype=torch.int32, device=dev),
                                           torch.tensor([0, n // ps], dtype=torch.int32, device=dev), None, ckv_scale, kpe_scale, check=True)
    packed, sf8 = O.quantize_ckv(ckv.float().numpy(), ckv_scale)
    k8 = O.quantize_kpe(kpe.float().numpy(), kpe_scale)
    assert np.array_equal(caches[1].view(torch.uint8).cpu().numpy().reshape(n, 32), sf8.reshape(n, 32))
    assert np.array_equal(caches[0].cpu().numpy().reshape(n, 256), packed.reshape(n, 256))
    assert np.array_equal(caches[2].view(torch.uint8).cpu().numpy().reshape(n, 64), k8.reshape(n, 64))
