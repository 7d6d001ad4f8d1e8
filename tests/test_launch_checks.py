"""What is decided before a launch: arguments that are refused (plain integers stand for device pointers, so no GPU is needed, and
where one is there, nothing is launched) and choices by size."""
import pytest

from omegalax_b200.ops import lib

A = 1 << 20      # an aligned address that is never read


@pytest.mark.parametrize("h,out,D,code", [(A + 2, A, 64, 6002), (A, A + 8, 64, 6002), (A, A, 60, 6001)])
def test_row_gather_of_the_head_wants_16_byte_rows(h, out, D, code):
    """A contiguous view may start anywhere; the gather reads 16 bytes at a time, as the products it stands before do."""
    assert lib.load().ob_ce_gather(h, A, A, out, 128, D, None) == code


@pytest.mark.parametrize("batch,rows,H,G,hd,causal,least,most", [
    (7, 512, 32, 8, 128, True, 1, 1), (4, 800, 32, 8, 128, True, 1, 1), (7, 512, 32, 4, 128, False, 1, 1), (2, 1000, 16, 8, 128, False, 1, 1),
    (1, 4096, 32, 8, 128, True, 1, 1), (2, 4096, 32, 8, 128, True, 1, 1), (1, 128, 16, 8, 128, True, 1, 1),
    (1, 4096, 32, 4, 128, True, 2, 4), (1, 3001, 32, 2, 256, True, 4, 8), (1, 512, 64, 4, 128, False, 8, 8), (1, 1000, 16, 8, 128, True, 2, 2)])
def test_ctas_share_a_key_tile_only_where_that_saves(batch, rows, H, G, hd, causal, least, most):
    """Sizes at which sharing was measured to lose, and to win by the factors named in ``attn_bwd_splits``."""
    from omegalax_b200.ops import kernels as K

    tiles = min(-(-rows // 128) * batch, batch * rows // 128 + batch) * (hd // 128)
    assert least <= K.attn_bwd_splits(tiles, H, G, -(-rows // 64), causal, batch * rows * G * hd) <= most


@pytest.mark.parametrize("M,N,K,few", [(1, 8, 64, True), (64, 4096, 32, True), (65, 4096, 512, False), (2048, 1024, 768, False), (500, 6144, 768, True),
                                       (2048, 1024, 1024, True), (1000, 6144, 4096, False), (128, 151936, 4096, True)])
def test_products_of_few_rows_go_where_they_are_faster(M, N, K, few):
    from omegalax_b200.ops import kernels

    assert kernels._use_few(M, N, K) is few


@pytest.mark.parametrize("rows,tiles,chunk", [(8192, 4, 4096), (32768, 4, 8192), (16384, 16, 1024), (4096, 64, 1024), (3000, 8, 4096),
                                              (2559, 4, 1024), (100, 8, 1024), (24000, 12, 2000)])
def test_more_tiles_than_the_default_bound_the_memory_of_the_head(rows, tiles, chunk):
    from omegalax_b200.trainers.loss import chunk_rows

    assert chunk_rows(rows, tiles) == chunk


def test_launch_module_converts_arguments_as_ctypes_does(monkeypatch):
    """Calls that the launchers answer on the host: same code, same kind of error, for numbers of each type and for what only
    ctypes takes."""
    import ctypes

    from omegalax_b200.ops import lib

    if not lib.available():
        pytest.skip("no library")
    lib.load()
    if lib._launch is None:
        pytest.skip("no C++ compiler or no headers of Python")
    fast = lib._launch
    buf = (ctypes.c_char * 16)()
    cases = [("ob_gemm_few", (None, 0, 0, None, True, 1, 0, 8, 8, 1 << 40, 0, 0, None, 0, None, 0)),     # a size of zero
             ("ob_gemm_few", (None, 0, 0, None, 1 << 32, 1, 8, 8, 8, 8, 0, 0, None, 0, None, 0)),        # rows cut to 32 bits: none
             ("ob_gemm_few", (None, 0, 0, None, 1, 1, 8, 7, 8, 8, 0, 0, None, 0, None, 0)),              # a pitch refused
             ("ob_gemm_few", (buf, 0, 0, None, 1, 1, 8, 7, 8, 8, 0, 0, None, 0, None, 0)),               # a pointer as an object
             ("ob_gemm_step", (8, 16, 16, None, 1, 8, 8, 8, 8, 8, 8, None, None, 1, None, 0, None, 0)),  # an int for a float
             ("ob_gemm_few", (1, 2)), ("ob_gemm_few", (None, 0, 0, None, 1.5, 1, 8, 8, 8, 8, 0, 0, None, 0, None, 0))]
    for name, args in cases:
        seen = []
        for call in (fast, None):
            monkeypatch.setattr(lib, "_launch", call)
            try:
                seen.append(lib.call(name, *args))
            except Exception as e:
                seen.append((type(e), str(e)))
        assert seen[0] == seen[1], (name, args, seen)
    assert fast("ob_gemm_few", *cases[2][1]) == 6001 and fast(*[cases[3][0], *cases[3][1]]) is None and fast("ob_unknown", 1) is None


@pytest.mark.parametrize("N,K,made", [(64, 128, False), (60, 128, True), (64, 100, True), (60, 100, True), (64, 128, True)])
def test_products_read_ahead_what_no_kernel_of_a_step_writes(monkeypatch, N, K, made):
    """Weights that a call pads, or that are no parameters, are read when the kernel before has ended."""
    import torch

    from omegalax_b200.ops import kernels, serving

    seen = []
    monkeypatch.setattr(kernels, "_call", lambda name, *args: seen.append((name, args)))
    monkeypatch.setattr(lib, "status_tensor", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(lib, "stream_ptr", lambda: 0)
    monkeypatch.setattr(serving, "_same", lambda *ts: 0)
    x, w = torch.zeros(3, K, dtype=torch.bfloat16), torch.nn.Parameter(torch.zeros(N, K, dtype=torch.bfloat16))
    if made and N % 8 == K % 8 == 0:
        w = w * 2
    with torch.no_grad():
        serving.project(x, w)
        serving.project(x, w, into=torch.zeros(3, N))
        if K % 8 == 0:
            kernels.gemm_step(x, w, act=2)
            kernels.gemm_relu_sq(x, w)
    flags = [args[{"ob_gemm_few": 11, "ob_gemm_step": 15}[name]] & 4 for name, args in seen]
    # a step's product is called with the weights as they are
    want = [0 if made else 4] * 2 + [4 if isinstance(w, torch.nn.Parameter) else 0] * (2 if K % 8 == 0 else 0)
    assert flags == want


def test_a_group_of_kernels_answers_for_itself(monkeypatch, tmp_path):
    """With one group loaded and no complete library, a prompt's squared ReLU asks that group which tiles fit."""
    import torch

    from omegalax_b200.ops import build, kernels

    if not lib.available():
        pytest.skip("no library")
    assert {"gemm_pair_sm100", "gemm_pair_wide_sm100"} <= set(build.GROUPS["latent_serving"])
    lib.load()
    monkeypatch.setattr(lib, "_partial", True)
    monkeypatch.setattr(lib, "LIB_PATH", tmp_path / "none.so")
    monkeypatch.setenv("OMEGALAX_B200_NO_BUILD", "1")
    seen = []
    monkeypatch.setattr(kernels, "_call", lambda name, *args: seen.append(name))
    monkeypatch.setattr(lib, "status_tensor", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(lib, "stream_ptr", lambda: 0)
    y = kernels.gemm_relu_sq(torch.zeros(8192, 256, dtype=torch.bfloat16), torch.zeros(4864, 256, dtype=torch.bfloat16))
    assert y.shape == (8192, 4864) and seen == ["ob_gemm_relu_sq"]


@pytest.mark.parametrize("trouble", ["compiler fails", "compiler is missing", "tree is read-only"])
def test_without_the_launch_module_the_library_loads_all_the_same(monkeypatch, tmp_path, trouble):
    """Where the module cannot be built, launchers are called through ctypes; to build it is an error only for who asks for that."""
    from omegalax_b200.ops import build

    if not lib.available():
        pytest.skip("no library")
    monkeypatch.delenv("OMEGALAX_B200_NO_BUILD", raising=False)
    monkeypatch.setenv("CXX", {"compiler fails": "/bin/false", "compiler is missing": str(tmp_path / "none"), "tree is read-only": "g++"}[trouble])
    monkeypatch.setattr(build, "launch_module", lambda: tmp_path / "_launch.so")
    monkeypatch.setattr(build, "BUILD", tmp_path / "build")
    if trouble == "tree is read-only":
        (tmp_path / "build").write_text("no folder can be made here")
    monkeypatch.setattr(lib, "_lib", None)
    monkeypatch.setattr(lib, "_launch", None)
    with pytest.warns(RuntimeWarning, match="ctypes"):
        lib.load()
    assert lib._launch is None
    with pytest.raises(lib.KernelError, match="6001"):
        lib.call("ob_gemm_few", None, 0, 0, None, 1, 1, 8, 7, 8, 8, 0, 0, None, 0, None, 0)
    with pytest.raises((OSError, RuntimeError)):
        lib.build_launch_module()


def test_the_compiler_of_the_launch_module_may_have_arguments(monkeypatch, tmp_path):
    import os
    import shutil
    import sysconfig

    from omegalax_b200.ops import build

    if not shutil.which("g++") or not os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")):
        pytest.skip("no C++ compiler or no headers of Python")
    monkeypatch.setenv("CXX", "env g++")
    monkeypatch.setattr(build, "launch_module", lambda: tmp_path / "_launch.so")
    monkeypatch.setattr(build, "BUILD", tmp_path / "build")
    lib.build_launch_module()
    assert (tmp_path / "_launch.so").exists() and build.launch_stamp().read_text() == lib._launch_table()[1]


def test_kernels_that_may_overlap_wait_for_the_one_before():
    """Every kernel whose launch takes the overlap of a recorded step: one without the wait reads what is not there yet, and the ones behind it
    no longer know that all before them have ended."""
    import re

    from omegalax_b200.ops import build

    launched, bodies = set(), {}
    for path in sorted(build.CSRC.glob("*.cu")) + sorted(build.CSRC.glob("*.cuh")):
        text = path.read_text()
        calls = re.findall(r"(?:OB_LAUNCH|[ =:)]launch)\(\(*(\w+)", text)
        launched |= {c for c in calls if c.endswith("_kernel")}
        if "kern" in calls:
            launched |= set(re.findall(r"auto kern = (\w+)", text))
        for m in re.finditer(r"__global__ void[^;{]*?(\w+_kernel)\(", text):
            bodies[m[1]] = text[m.end():text.index("\n}\n", m.end())]
    assert len(launched) > 25 and {"column_sum_kernel", "gemm_few_kernel", "decode_rows_kernel", "experts_few_kernel", "paged_decode_kernel"} <= launched
    assert [k for k in sorted(launched) if not re.search(r"grid_(begin|wait)\(\)", bodies[k])] == []
