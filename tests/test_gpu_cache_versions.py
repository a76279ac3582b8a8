"""Saved tuning files: the projectors' numbers of a version 3 file stood for other
launch shapes, so that such a file gives them the built-in ones."""
import pytest

from test_gpu_sart import make_case

pytestmark = pytest.mark.gpu


def test_projector_shapes_of_an_earlier_version_are_not_taken(torch_cuda, oracle, tmp_path):
    import mcsart_b200 as m
    torch = torch_cuda
    g, it, img0, proj, F = make_case(oracle, motion=False, op_iter=(1,), seed=3)
    saved, old, bare = tmp_path / "s.txt", tmp_path / "old.txt", tmp_path / "bare.txt"
    with m.Context(0, stream=torch.cuda.current_stream().cuda_stream) as c:
        c.autotune(geo=g, n_views=it["n_views"], lambda_=1.0, angles=it["angles"],
                   volumes=it["volumes"], flows=it["flows"], img=torch.zeros(img0.shape, device="cuda"),
                   proj=torch.as_tensor(proj).cuda(), options=m.default_options())
        best = c.tuning_get(g)
        c.tuning_save(saved)
    key = [ln.split()[0] for ln in saved.read_text().splitlines() if not ln.startswith("#")][0]
    old.write_text(f"# mcsart tuning cache v3: key fp1 fp3 bp warp fup\n{key} 2 1 3 2 1\n")
    bare.write_text(f"{key} 2 1 3 2 1\n")
    for path, want in ((saved, best), (old, [-1, -1, 3, 2, 1]), (bare, [2, 1, 3, 2, 1])):
        with m.Context(0, stream=torch.cuda.current_stream().cuda_stream) as c:
            assert c.tuning_load(path) == 1
            assert c.tuning_get(g) == list(want)
