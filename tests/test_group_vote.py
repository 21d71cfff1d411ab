"""What an epilogue group of the tile product does after a bounded wait gave up: all of its threads go on, or none.  A thread
that decided by its own look at the flag could leave the others waiting at the group's next barrier for good."""
import ctypes as C
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_role_branches_on_its_own_look_at_the_flag():
    src = open(os.path.join(HERE, "..", "cnet_b200", "csrc", "cgemm_tc.cu")).read()
    kernel = src[src.index("\ncgemm_tc_k("):src.index("__global__", src.index("\ncgemm_tc_k("))]
    roles, ends = kernel.rsplit("finish();", 1)              # behind the roles' common end nothing sets the flag any more
    assert "cluster_reduce<2" in ends
    looks = [line.strip() for line in roles.splitlines() if re.search(r"\*\s*abort_flag\b(?!\s*=)", line)]
    looks = [line for line in looks if not line.startswith("volatile int* abort_flag")]
    assert looks == [], looks
    assert roles.count("epi_gave_up(group, abort_flag)") == 3


@pytest.mark.gpu
def test_a_group_gives_one_answer(tmp_path):
    import torch
    so = str(tmp_path / "vote.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared",
                    os.path.join(HERE, "cpp", "group_vote_probe.cu"), "-o", so], check=True,
                   env={**os.environ, "PATH": os.environ.get("PATH", "") + ":/usr/local/cuda/bin"})
    votes = [(0, 0)] + [(1 << t, 0) for t in (0, 31, 32, 64, 127)] + [(0, 1 << t) for t in (1, 63, 96)] + [((1 << 128) - 1, 1 << 77), (0, 0)]
    words = [[(v >> (32 * i)) & 0xffffffff for i in range(4)] for pair in votes for v in pair]
    yes = torch.tensor(words, dtype=torch.int64).to(torch.int32).cuda()
    out = torch.full((len(votes) * 2, 128), 9, dtype=torch.uint8, device="cuda")
    assert C.CDLL(so).vote(C.c_void_p(yes.data_ptr()), len(votes), C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = torch.tensor([[int(v != 0)] * 128 for pair in votes for v in pair], dtype=torch.uint8)
    assert torch.equal(out.cpu(), want)
