"""The C ABI without a GPU: the library loads, exports every declared symbol,
and rejects bad arguments before touching the device."""
import re
from pathlib import Path

from token2tile_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent


def declared_symbols():
    text = (ROOT / "include" / "t2t_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(t2t_\w+)\s*\(", text)))


def test_library_exports_every_declared_symbol(lib):
    names = declared_symbols()
    assert len(names) >= 19
    for n in names:
        assert hasattr(lib, n), n
    assert set(_lib.SIGNATURES) == set(names)
    assert lib.t2t_version() >= 100


def test_workspace_sizes_are_pure_host_functions(lib):
    assert lib.t2t_kmeans_maintain_ws_bytes(40, 75600, 512, 2048) > 40 * 75600 * 4
    assert lib.t2t_vstats_gather_ws_bytes(40, 2048) >= 40 * 2048 * 128 * 4
    assert lib.t2t_tile_attn_ws_bytes(2, 4096) >= 2 * 4096 * (256 + 4)
    ints = lib.t2t_tile_attn_plan_ints(40, 75600, 512)
    assert ints >= 40 * 2049 + 4 * 40 * (512 + 75600 // 256) + 40 * 512
    assert lib.t2t_centroid_update_ws_bytes(2, 4096, 2048) > 0
    assert lib.t2t_assign_ws_bytes(40, 75600) == 4


def test_grouping_takes_few_histograms_where_their_sums_are_what_takes_long(lib):
    """256 rows per histogram while a thread that adds them up meets at most 64 (once per 1024 clusters), 1024 beyond."""
    def histograms(H, N, Cn):
        rest = H * Cn * 4 + H * N * 4               # cluster bases and the permutation, both multiples of 256 bytes here
        return (lib.t2t_centroid_update_ws_bytes(H, N, Cn) - rest) // (H * Cn * 4)

    assert [histograms(1, N, 2048) for N in (4096, 8192, 16384, 65536)] == [16, 32, 16, 64]
    assert [histograms(40, N, 512) for N in (4096, 16384, 32768)] == [16, 64, 32]


def test_null_and_bad_arguments_are_rejected(lib):
    assert lib.t2t_project(0, 0, 0, 1, 1, 0, 0) == 1
    assert lib.t2t_assign(0, 0, 0, 2, 4096, 32, -1, 0, 0, 0, 0, 0) == 1
    assert lib.t2t_assign_exact(0, 0, 0, 2, 4096, 32, -1, 0, 0) == 1
    assert lib.t2t_gather_rows(0, 0, 0, 2, 4096, 0) == 1
    assert lib.t2t_score_select_union(0, 0, 0, 0, 0, 0, 0, 0, 2, 4096, 32, 0, 0, 0, 0, 0) == 1
    assert lib.t2t_score_select_union_exact(0, 0, 0, 0, 0, 0, 0, 0, 2, 4096, 32, 0, 0) == 1
    assert lib.t2t_vstats_gather(0, 0, 0, 0, 0, 0, 2, 4096, 2048, 0, 0, 0) == 1
    assert lib.t2t_tile_attn_plan(0, 0, 0, 0, 2, 4096, 32, 0) == 1
    assert lib.t2t_umma_selftest(0, 0, 0, 0, 0, 0, 0) == 1
    assert lib.t2t_gather4_selftest(0, 0, 0, 0, 0, 0) == 1
    assert lib.t2t_wait_timeout_selftest(0, 0, 0) == 1
    assert lib.t2t_softmax_give_up_selftest(0, 0, 0, 0, 0, 0, 0) == 1
    assert lib.t2t_select_give_up_selftest(0, 0, 0, 0) == 1
    assert lib.t2t_rotation_selftest(0, 0, 1, 0) == 1


def test_kernels_built_with_other_register_counts_are_refused(lib):
    """The attention kernels' warps trade registers out of 128 a thread; registers are allocated in eights."""
    assert [lib.t2t_register_split_selftest(r) for r in (128, 121)] == [0, 0]
    assert [lib.t2t_register_split_selftest(r) for r in (0, 64, 104, 120, 129, 255)] == [2] * 6


def test_readers_of_a_shared_task_release_it_at_cluster_scope():
    """The other CTA of a pair overwrites a task's slot behind the TFREE barrier.  No run can show a missing order, so the
    source is read: every arrival there is a release at cluster scope, the wait in front of the stores an acquire."""
    text = (ROOT / "token2tile_b200" / "csrc" / "tile_attn.cu").read_text()
    pair = text[text.index("attn2_kernel("):text.index("exact attention, tasks of at most QT rows")]
    role = text[text.index("void softmax_role("):text.index("attn2_kernel(")]
    arrivals = re.findall(r"(mbar_\w+|arrive)\([^;]*\btfree\b", role + pair)
    assert len(arrivals) >= 4 and set(arrivals) == {"mbar_release_peer"}
    assert re.findall(r"(mbar_wait\w*)\(bars \+ B_TFREE", pair) == ["mbar_wait_warp_cluster"]


def test_operator_dir_points_at_the_sources():
    import token2tile_b200
    d = Path(token2tile_b200.operator_dir())
    assert (d / "deploy_step.py").exists() and (d / "csrc" / "tile_attn.cu").exists()
