"""How products are cut, from their sizes alone: no GPU."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as ge
    ge.build()
    from mesh_transformer import _lib
    return _lib


def _handle(lib, **kw):
    base = dict(layers=2, d_model=4096, n_heads=16, n_vocab=50400, pe_rotary_dims=64, seq=2048, cores_per_replica=1, rank=0,
                max_batch=1, max_gen=8, max_rows=2048)
    base.update(kw)
    h = ctypes.c_void_p()
    lib.check(lib.lib.mtj_create(ctypes.byref(lib.MtjConfig(**base)), ctypes.byref(h)))
    return h


@pytest.mark.parametrize("sizes", [dict(), dict(cores_per_replica=2), dict(cores_per_replica=4), dict(cores_per_replica=8),
                                   dict(d_model=8448, n_heads=33)])
def test_short_prompts_keep_the_gpu_busy_in_the_output_projection(lib, sizes):
    """33 to 192 rows are one tile high: whole K would keep d / 256 of the 74 block pairs busy (16 at width 4096), whether the
    sum is fused with the norm behind it (one GPU, rows up to 8192 wide) or not."""
    h = _handle(lib, **sizes)
    d = sizes.get("d_model", 4096)
    for rows in (33, 56, 64, 65, 128, 129, 192):
        pieces = lib.lib.mtj_k_out_projection_pieces(h, rows, 0)
        assert 2 <= pieces <= 8, (rows, pieces)
        assert (d + 255) // 256 * pieces >= 32, (rows, pieces)
    lib.lib.mtj_destroy(h)


def test_evaluation_keeps_whole_k_from_129_rows_on(lib):
    h = _handle(lib)
    assert [lib.lib.mtj_k_out_projection_pieces(h, rows, 1) for rows in (33, 128, 129, 192, 193, 700, 2048)] == [8, 8, 1, 1, 1, 1, 1]
    assert lib.lib.mtj_k_out_projection_pieces(h, 0, 0) < 0
    lib.lib.mtj_destroy(h)


def test_the_pair_mask_reaches_the_output_projection(lib, monkeypatch):
    """Only block pairs cut K: with them switched off at that call site its K stays whole."""
    for mask, whole in (("7", False), ("5", True), ("2", False), ("0", True)):
        monkeypatch.setenv("MTJ_TC_PAIR", mask)
        h = _handle(lib)
        assert (lib.lib.mtj_k_out_projection_pieces(h, 136, 0) == 1) == whole, mask
        lib.lib.mtj_destroy(h)


def _workspace(lib, h):
    n = lib.lib.mtj_workspace_bytes(h)
    lib.lib.mtj_destroy(h)
    return n


def test_the_workspace_follows_the_model(lib):
    """The scratch of products cut along K is what the model's own sizes can ask for: a small model does not pay for a large one's."""
    from mesh_transformer import registry
    from tests import stack_util as su
    small = _handle(lib, d_model=256, n_heads=4, n_vocab=512, pe_rotary_dims=16, seq=128, max_batch=2, max_rows=128)
    assert _workspace(lib, small) < 8 << 20
    sizes = {}
    for dtype in ("float32", "bfloat16"):
        for name, cfg in (("keselix", su.model([su.attn(ff=44)])), ("bavutar", su.bavutar([su.gqa()]))):
            cfg = registry.prepare(dict(cfg, mtj_dtype=dtype, seq=128))
            h = ctypes.c_void_p()
            caps = dict(rank=0, max_batch=1, max_gen=1, max_rows=128, hilo_max_batch=0, mega_max_batch=0, tc_decode_min_batch=0, wait_limit=0)
            lib.check(registry.family(cfg).create(cfg, caps, ctypes.byref(h)))
            sizes[dtype, name] = _workspace(lib, h)
    assert max(sizes.values()) < 8 << 20, sizes
