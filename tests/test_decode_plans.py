"""The few-token kernels' plans, without a device: a grid of more CTAs than SMs is a second wave unless two of them fit an
SM's shared memory.  The second wave would stage all activations again, and the next kernel could not be set up beside the
first (decode_gemv.cu, decode_moe.cu)."""
import ctypes as C
import importlib
import random

import pytest

capi = importlib.import_module("jdm-ghassan_v1_flach_b200.capi")
SMS = 148                                      # what the library plans for without a device, and a B200's
SM_BYTES = 228 * 1024                          # shared memory of an SM
CTA_BYTES = 1024 + 256                         # the system's share of a CTA, and the kernels' static variables (rounded up)
KINDS = [0, 1, 2, 3]


@pytest.fixture(scope="module")
def so():
    return C.CDLL(capi.LIB_PATH)


def gemv_plan(so, kind, M, N, K, norm, plain=0):
    ctas, smem = C.c_int(), C.c_int()
    rc = so.b200_digit_gemv_plan(kind, M, N, K, norm, plain, C.byref(ctas), C.byref(smem))
    return rc, ctas.value, smem.value


def moe_plan(so, kind, M, d, E, ne, K, SH, alone=0):
    ctas, smem = (C.c_int * 3)(), (C.c_int * 3)()
    rc = so.b200_moe_digit_plan(kind, M, d, E, ne, K, SH, alone, ctas, smem)
    return rc, list(ctas), list(smem)


def one_wave(ctas, smem):
    per_sm = -(-ctas // SMS)
    return per_sm == 1 or per_sm * (smem + CTA_BYTES) <= SM_BYTES


# in_proj, q / k / v and out_proj of models 768 to 4096 wide, and generic sizes
SIZES = [(768, 3224), (1536, 6448), (3072, 1536), (2560, 10448), (4096, 16768), (4096, 6144), (8192, 4096), (256, 16), (1024, 100352),
         (2048, 8448), (5120, 20832)]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("K,N", SIZES)
def test_products_run_in_one_wave(so, kind, K, N):
    for M in range(1, 9):
        for norm, plain in ((0, 0), (1, 0), (0, 1)):
            rc, ctas, smem = gemv_plan(so, kind, M, N, K, norm, plain)
            if rc == 0:
                assert one_wave(ctas, smem), f"{M} tokens: {ctas} CTAs of {smem} bytes"


LAYERS = [(768, 512, 16, 2, 1024), (1536, 512, 64, 6, 1024), (2560, 512, 32, 4, 1024), (4096, 768, 72, 10, 1536), (1536, 1024, 32, 8, 2048),
          (1536, 512, 64, 6, 0)]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("d,E,ne,K,SH", LAYERS)
def test_moe_layers_run_in_one_wave(so, kind, d, E, ne, K, SH):
    for M in range(1, 9):
        for alone in (0, 1):
            rc, ctas, smem = moe_plan(so, kind, M, d, E, ne, K, SH, alone)
            if rc == 0:
                for k in range(3):
                    assert one_wave(ctas[k], smem[k]), f"{M} tokens, kernel {k + 1}: {ctas[k]} CTAs of {smem[k]} bytes"


# in_proj and the layer of the H-Tiny shape: two CTAs fit, so the grid is doubled from three (two) tokens on
def test_two_ctas_where_they_fit(so):
    for M in range(1, 9):
        assert gemv_plan(so, 3, M, 6448, 1536, 1)[1] == (148 if M <= 2 else 296)
        rc, ctas, _ = moe_plan(so, 3, M, 1536, 512, 64, 6, 1024)
        assert rc == 0 and ctas[1] == (148 if M == 1 else 296 // M * M)


# By itself a product keeps one CTA an SM where its share is one set in half an SM.
def test_products_by_themselves(so):
    for M in range(3, 9):
        for K, N, two in [(768, 3224, False), (1536, 6448, False), (512, 24000, True), (2560, 10448, M <= 4)]:
            rc, ctas, smem = gemv_plan(so, 3, M, N, K, 0, 1)
            assert rc == 0 and ctas == (296 if two else 148), (M, K, N, ctas)
            assert two or smem <= SM_BYTES // 2 or K == 2560


# A MoE layer by itself: the second CTA only for gate / up of seven products of a chunk and more, and for down whose three tiles
# and more do not fit half an SM.
def test_layers_by_themselves(so):
    def ctas(*a):
        rc, c, _ = moe_plan(so, *a)
        assert rc == 0
        return c
    for alone, gate_up in ((0, 256), (1, 148)):
        assert ctas(3, 2, 768, 512, 16, 2, 1024, alone)[1] == gate_up
    assert ctas(3, 3, 768, 512, 16, 2, 1024, 1)[1] == 98 * 3
    for alone, down in ((0, 296), (1, 148)):
        assert ctas(3, 2, 4096, 256, 8, 2, 1536, alone)[2] == down
        assert ctas(3, 8, 768, 512, 16, 2, 1024, alone)[2] == (37 if not alone else 18) * 8
        assert ctas(3, 3, 2560, 512, 32, 4, 1024, alone)[2] == 98 * 3


def test_random_shapes_run_in_one_wave(so):
    r = random.Random(1)
    for _ in range(400):
        kind, M = r.choice(KINDS), r.randint(1, 8)
        K, N = 256 * r.randint(1, 40), 16 * r.randint(1, 1200)
        norm = r.randint(0, 1)
        rc, ctas, smem = gemv_plan(so, kind, M, N, K, norm, 0 if norm else r.randint(0, 1))
        assert rc != 0 or one_wave(ctas, smem), (kind, M, N, K, ctas, smem)
        args = (kind, M, 256 * r.randint(1, 20), 256 * r.randint(1, 6), 8 * r.randint(2, 16), r.randint(1, 12), 256 * r.randint(0, 8))
        rc, ctas, smem = moe_plan(so, *args, r.randint(0, 1))
        assert rc != 0 or all(one_wave(c, s) for c, s in zip(ctas, smem)), (args, ctas, smem)
