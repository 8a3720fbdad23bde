"""The division sequence for fixed divisors over the lengths the pair forms take (CPU)."""
import subprocess

from conftest import REPO


def test_every_length_and_its_square(tmp_path):
    exe = tmp_path / "fixed_div_range"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", str(REPO / "tests" / "cpp" / "fixed_div_range.c"),
                    "-o", str(exe), "-lm"], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    ok, divisors, tested = out.stdout.split()
    assert ok == "ok" and int(divisors) >= 80 and int(tested) >= 60 * (1 << 17)
