"""with_split(): the split of an operator's rows over threads, and whole rows where
the caller asks for them (reorthogonalisation runs on whole rows alone)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_split_and_whole_rows(tmp_path):
    exe = str(tmp_path / "split_check")
    cmd = [os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "--extended-lambda", "-gencode",
           "arch=compute_100a,code=sm_100a", "-diag-suppress", "177,550", "-I", os.path.join(ROOT, "include"), "-I",
           os.path.join(ROOT, "qmbcuda_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "split_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout
    got = {}
    for line in out.splitlines():
        name, n, s, whole = line.split()
        assert whole == "1", line
        got[name, int(n)] = int(s)
    assert len(got) == 78
    for (name, n), s in got.items():
        want = {"sell": 4 if n < 16384 else 2 if n < 300000 else 1, "sell_c64": 4 if n < 16384 else 2 if n < 640000 else 1,
                "mf": 8 if n < 16384 else 4 if n < 131072 else 2 if n < 400000 else 1,
                "mf_no_group": 8 if n < 16384 else 4 if n < 40000 else 2 if n < 131072 else 1, "ref_ell": 4, "coded": 1}[name]
        assert s == want, (name, n, s)
