"""A decode on a system whose driver builds no tensor maps runs the CUDA-core kernel, which knows no clusters.

``decode_fallback_check.cpp`` calls the built library over a stand-in for the CUDA runtime, so this needs no GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    from rustorch_b200 import build
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    exe = str(tmp_path_factory.mktemp("decode_fallback") / "check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-rdynamic", "-isystem", os.path.join(cuda, "include"), "-o", exe,
                    os.path.join(HERE, "decode_fallback_check.cpp"), "-ldl"], check=True, capture_output=True, text=True)

    def run(**overrides):
        env = {k: v for k, v in os.environ.items() if not k.startswith("RT_ATTN_")}
        r = subprocess.run([exe, build.build()], env={**env, **overrides}, capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
        return r.stdout.splitlines()
    return run


def test_launches_are_those_without_clusters(launches):
    """Chunks within the scratch, and the launch that merges them, for the plain call, the pushed record and the exchange."""
    without = launches(RT_ATTN_DECODE_CLUSTER="0")
    assert without.count("status 0 0 0") == 5 and all(" cluster 1 " in x for x in without if x.startswith("grid"))
    assert launches() == without
    for size in ("2", "16"):
        assert launches(RT_ATTN_DECODE_CLUSTER=size) == without
