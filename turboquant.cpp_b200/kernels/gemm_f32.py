"""True float32 products of many tokens on the tensor cores, operands as three bfloat16 values each (csrc/gemm_f32.cu)."""
from __future__ import annotations

from ctypes import c_int, c_longlong, c_void_p
from functools import lru_cache
from typing import Optional

import torch

from ..csrc.build import load_kernel
from ._call import KernelError, check, ptr, stream
from .gemm_tc import status_word

_LIB = "gemm_f32"
MIN_TOKENS = 9
# Results from which on this kernel is ahead of the library's fp32 product.  It takes some 18 us per 1,000 elements of K whatever there
# is to do up to a GPU full of tiles, the library's time grows from the first tile on.  us, here / library, K 2,048: 41 / 38 at 64
# tokens x 2,048, 41 / 42 at 96, 42 / 57 at 192, 47 / 145 at 700; 41 / 41 at 17 x 6,144, 42 / 54 at 33, 79 / 309 at 700; 41 / 38 at 128 x
# 1,024, 41 / 42 at 192.  K 512: 15 / 13 at 64 x 2,048, 15 / 19 at 192.  K 5,632: 101 / 95 at 64 x 2,048, 102 / 105 at 128.
MIN_RESULTS = 200_000
# Below this a product is a few launches' time either way.
MIN_K = 64
# Sums shorter than LONG_K of FEW_TOKENS or fewer are the library's: the tiles' setting up is more than what they compute.  us, here / library:
# K 64, 40,960 rows 16 / 11 at 16 tokens, 19 / 17 at 64, 20 / 21 at 65; K 128, 20,480 rows 14 / 12 at 32, 16 / 20 at 65, 40,960 rows 20 / 15 at
# 16, 24 / 31 at 65; K 512, 20,480 rows 26 / 27 at 16, 30 / 41 at 64.  Few weight rows are no reason: 4,096 tokens, K 64, 64 rows 15 / 15, K
# 512 16 / 15, K 2,048 44 / 42, K 5,632 130 / 139.
LONG_K, FEW_TOKENS = 256, 64


@lru_cache(maxsize=None)
def runs() -> bool:
    """Whether the library on hand can launch the kernel: its warpgroups share out the registers that this repository's compiler gives
    it, and another compiler may give it fewer."""
    return bool(load_kernel(_LIB).tq_gemm_f32_runs())


def pays(x: torch.Tensor, w: torch.Tensor) -> bool:
    """float32 x [T, K] (rows on 16-byte boundaries) and w [N, K] that this kernel takes and is the faster one for."""
    T, K = x.shape
    return (T >= MIN_TOKENS and T * w.shape[0] >= MIN_RESULTS and K % 4 == 0 and K >= MIN_K and (K >= LONG_K or T > FEW_TOKENS)
            and x.dtype == torch.float32 and w.dtype == torch.float32
            and w.dim() == 2 and w.shape[1] == K and w.is_contiguous() and x.stride(1) == 1 and x.stride(0) % 4 == 0 and x.stride(0) >= K
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and x.device == w.device and x.device.index == torch.cuda.current_device()
            and not (torch.is_grad_enabled() and (x.requires_grad or w.requires_grad)) and runs())


def gemm_f32(x: torch.Tensor, w: torch.Tensor, tokens: int = 0, status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """x [T, K] (rows any multiple of four floats apart) times w [N, K] transposed -> [T, N] in float32; as accurate as a float32 sum.
    tokens: of a tile (0: the launcher's choice)."""
    (T, K), N = x.shape, w.shape[0]
    if x.dtype != torch.float32 or w.dtype != torch.float32 or w.shape[1] != K or not x.is_cuda or x.stride(1) != 1:
        raise KernelError("gemm_f32: float32 CUDA tensors x [T, K] and w [N, K] with dense rows")
    out = torch.empty((T, N), dtype=torch.float32, device=x.device)
    lib = load_kernel(_LIB)
    check(_LIB, lib.tq_gemm_f32(c_void_p(x.data_ptr()), c_longlong(x.stride(0)), ptr(w), ptr(out), c_int(T), c_int(N), c_int(K), c_int(tokens),
                                ptr(status if status is not None else status_word(x.device)), stream()))
    return out
