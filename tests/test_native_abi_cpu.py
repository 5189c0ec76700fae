"""Layout agreement between the ctypes mirrors and the structures compiled into the kernel library, and the host-only
planning entry points.  None of this launches a kernel, so it runs wherever the library loads (a box without a GPU
included); it catches a field added on one side only before any launch reads a shifted pointer."""
import ctypes as C
import os

import pytest

from smcsd_b200.ops import native as K

_LIB = os.path.join(os.path.dirname(K.__file__), "libsmcsd_b200.so")
pytestmark = pytest.mark.skipif(not os.path.exists(_LIB), reason="kernel library not built")


def test_structure_sizes_match_the_library():
    from smcsd_b200.ops.native_forward import PfParams
    from smcsd_b200.parallel.particle_parallel import PpLocal, PpWorld
    L = K.lib()
    pairs = [(K.SlotArrays, "smc_slot_arrays_size"), (K.CycleIO, "smc_cycle_io_size"), (K.TpLink, "smc_tp_link_size"),
             (K.TpPeers, "smc_tp_peers_size"), (PpWorld, "smc_pp_world_size"), (PpLocal, "smc_pp_local_size"),
             (PfParams, "smc_pf_params_size")]
    for cls, fn in pairs:
        f = getattr(L, fn)
        f.restype = C.c_int
        assert C.sizeof(cls) == f(), f"{cls.__name__} differs from the compiled structure"


def test_split_plans_are_bounded_and_monotone():
    """Key-range split counts of the attention launches: at least one, never more than the cluster limit, and not
    shrinking as the context grows (a plan that shrank would re-key the captured cycle graph back and forth)."""
    prev = 0
    for keys in (64, 256, 1024, 4096, 16384, 65536):
        ks = K.attention_tc_splits(4, 8, keys, 128)
        assert 1 <= ks <= 16 and ks >= prev
        prev = ks
    # more sequences or heads fill the GPU by themselves: fewer splits are planned, never more
    assert K.attention_tc_splits(64, 8, 16384, 128) <= K.attention_tc_splits(1, 8, 16384, 128)


def test_layered_structures_match_the_library():
    """Sizes are asserted when the layered entry points are declared; the split planner stays within the cluster limit."""
    K.layered_lib()
    for tiles in (1, 8, 37, 200):
        prev = 0
        for keys in (1, 64, 500, 4096, 65536):
            ks = K.latent_tc_splits(tiles, 256, keys)
            assert 1 <= ks <= 8 and ks >= prev and (ks == 1 or tiles * ks <= 148)
            prev = ks


def test_kernels_that_wait_for_an_earlier_one_read_it_through_plain_pointers():
    """Loads through ``const T* __restrict__`` parameters count as invariant: the compiler may move them above griddepcontrol.wait, ahead of
    the kernel that writes what they read.  Tables and weights, which no kernel writes, may have the qualifier."""
    import re
    fixed = {"w", "embed", "rope"}
    csrc = os.path.join(os.path.dirname(K.__file__), "csrc")
    text = open(os.path.join(csrc, "fused_ops.cu")).read()
    for kernel in ("add_rmsnorm_kernel", "rope_kv_write_vec_kernel"):
        params = re.search(r"__global__[^;{]*\b" + kernel + r"\(([^{]*)\)\s*\{", text).group(1)
        assert "pdl" in params
        assert set(re.findall(r"const \w+\* __restrict__ (\w+)", params)) <= fixed, kernel
    for name in ("attention_prompt_tc.cu", "gdn_chunk.cu", "gemm_wide.cu"):
        assert "__restrict__" not in open(os.path.join(csrc, name)).read(), name


@pytest.mark.parametrize("N,kdim,M,groups,rows16,wide", [
    (3072, 2048, 640, 1, False, True), (2048, 8192, 320, 1, False, False), (3072, 2048, 128, 1, False, False),
    # bf16 rows: half-empty pairs, one full round of small tiles, three blocks of K
    (128, 64, 1024, 32, True, False), (128, 64, 1024, 32, False, True), (64, 512, 4096, 8, True, False), (384, 256, 1024, 32, True, False),
    (2048, 256, 2048, 1, True, False), (2048, 256, 1024, 1, True, True), (2048, 4096, 2048, 1, True, True), (8192, 64, 1024, 1, True, False),
    (8192, 512, 4096, 1, True, True), (512, 512, 1408, 16, True, True)])
def test_which_products_take_cta_pairs(N, kdim, M, groups, rows16, wide):
    """Both sides of the borders, as they were measured."""
    assert (K.lib().smc_gemm_wide_tile(N, (kdim + 63) // 64, M, groups, int(rows16)) > 0) == wide


def test_prompt_kernels_refuse_addresses_that_their_wide_accesses_cannot_take():
    """Every pointer in turn off its border: refused on the host, ahead of any launch."""
    L, p = K.lib(), 1 << 20
    vp, i, f = C.c_void_p, C.c_int, C.c_float
    L.smc_attention_prompt_tc.argtypes = [vp, vp, i, vp, vp, i, vp, i, i, vp, i, vp, i, i, i, i, C.c_float, vp, i, vp]

    def attention(q=p, gate=None, k=p, v=p, tiles=p, out=p):
        return L.smc_attention_prompt_tc(q, gate, 64, k, v, 7, p, 8, 1, tiles, 1, out, 4, 4, 1, 64, 0.125, p, 0, None)
    for name in ("q", "k", "v", "tiles", "out"):
        assert attention(**{name: p + 8}) == -86, name
    assert attention(gate=p + 4) == -85
    L.smc_gdn_chunked.argtypes = [vp, vp, i, vp, vp, vp, vp, vp, vp, i, i, vp, vp, i, i, i, i, i, f, vp, i, vp, vp, i, vp]

    def delta(conv=p, proj=p, out=p, scratch=p):
        return L.smc_gdn_chunked(conv, proj, 1024, p, p, p, p, p, out, 1, 64, None, None, 64, 1, 1, 128, 128, 1e-6, scratch, 8, p, None, 0, None)
    assert delta(conv=p + 8) == delta(proj=p + 4) == delta(out=p + 4) == -105 and delta(scratch=p + 8) == -106
