"""Which form of a kernel a size takes: rules that run on the host, asked through the libraries themselves."""
import importlib
import random

import numpy as np
import pytest

SMS = 148


@pytest.fixture(scope="module")
def ops():
    return importlib.import_module("daisi-llogos_b200.kernels.ops")


@pytest.mark.parametrize("n,o,k", [(2621441, 128, 128), (2680889, 128, 128), (3343748, 100, 4), (3905846, 100, 128), (3987930, 128, 512),
                                   (64 * 65535, 128, 128)])
def test_float32_tiles_of_very_many_rows_fit_a_grid(ops, n, o, k):
    """64 rows a tile always fit up to 64 x 65,535 rows, the most that a product takes; lower tiles do not."""
    rows, _ = ops.gemm_simt_form(n, o, k, SMS)
    assert -(-n // rows) <= 65535


def test_float32_tiles_of_any_size(ops):
    rng = random.Random(5)
    for _ in range(20000):
        n, o, k = (int(2 ** rng.uniform(low, high)) for low, high in ((5.1, 21.99), (0, 17), (0, 14)))
        k = 4 * k
        rows, ranks = ops.gemm_simt_form(n, o, k, rng.choice((1, 16, 132, SMS)))
        assert rows in (40, 48, 56, 64) and ranks in (1, 2, 4) and -(-n // rows) <= 65535
        assert ranks == 1 or -(-k // 32) >= 2 * ranks           # every block of a tile has two steps or more, but for the last one's rest


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("parts", [2, 4, 8])
def test_blocks_that_share_a_tiles_keys_have_a_multiprocessor_each(ops, hd, parts):
    """Blocks of a cluster wait for one another with all of a multiprocessor's tensor memory in hand: two must not fit on one (228 KB of
    shared memory, 1 KB of it the system's for every block; at most 227 KB for a block)."""
    need = ops._lib("attention_tc").llg_attn_prefill_few_smem(hd, parts)
    assert 2 * (need + 1024) > 228 * 1024 and need <= 227 * 1024


def test_prompt_attention_goes_by_host_sizes_only_where_they_are_the_steps(ops):
    """The form for few long sequences has a grid made for the sizes on the host: with sizes that understate the step's queries rows would
    stay unwritten, so it is not taken (0: the other instance, which asks the device alone)."""
    sizes = np.asarray([(1083, 83), (900, 83)], dtype=np.int32)
    assert ops.attn_prefill_parts(sizes, 16, 4, 0, SMS, n_tokens=166) == ops.attn_prefill_parts(sizes, 16, 4, 0, SMS) == 4
    for n_tokens in (165, 167, 240):
        assert ops.attn_prefill_parts(sizes, 16, 4, 0, SMS, n_tokens=n_tokens) == 0


@pytest.mark.parametrize("n,o,k,rows,ranks", [
    (33, 200, 132, 40, 1), (63, 129, 1036, 40, 4), (100, 3170, 252, 40, 1), (65, 300, 288, 40, 4), (64, 128, 1036, 40, 4), (65, 257, 4104, 40, 4),
    (200, 300, 2052, 40, 4), (130, 24000, 64, 48, 1), (100, 3072, 2048, 40, 2), (88, 3396, 296, 48, 2), (163, 798, 240, 48, 4), (50, 12581, 36, 56, 1),
    (53, 5151, 564, 56, 2), (51, 2413, 304, 56, 4), (59, 9475, 56, 64, 1), (57, 19034, 180, 64, 2), (59, 2246, 300, 64, 4),
    (300, 4096, 4096, 64, 4), (448, 3072, 2048, 64, 4)])
def test_the_float32_tiles_that_sizes_take(ops, n, o, k, rows, ranks):
    """On 148 multiprocessors; the first ones are the sizes at which test_gemm_simt_float32_rows runs the product as it chooses by itself,
    the last two sizes where lower tiles are slower (339 us in tiles of 40 rows and 319; 170 and 163)."""
    assert ops.gemm_simt_form(n, o, k, SMS) == (rows, ranks)
