"""The integer conversions between double and double-float in the generated element kernels give
the bits of the FP64 formulas hi = (float)x, lo = (float)(x - hi) and hi + lo, or refuse (host build)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_conversions_equal_the_fp64_formulas(tmp_path):
    text = open(os.path.join(ROOT, "symx_gb300", "csrc", "df_convert.inl")).read().strip()
    assert text.startswith('R"(') and text.endswith(')"')
    (tmp_path / "df_convert.h").write_text(text[3:-2])
    exe = tmp_path / "test_df_convert_host"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(tmp_path),
                    os.path.join(ROOT, "tests", "cpp", "test_df_convert_host.cpp"), "-o", str(exe)], check=True)
    n, bad, refused = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert n > 10_000_000 and bad == 0 and refused < 0.7 * n
