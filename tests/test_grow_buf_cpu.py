"""The decoder's scratch over a fake allocator (csrc/grow_buf.h, host code):
memory that is refused to the scratch it can do without is no error, and that
scratch is given up where any other is refused."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_scratch_where_memory_is_short(tmp_path):
    exe = tmp_path / "grow_buf"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", f"-I{ROOT / 'bzip2gpu_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "grow_buf.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.stdout.strip() == "ok", f"check at line {r.stdout.strip()} of grow_buf.cpp"


def test_the_jumps_scratch_is_budgeted():
    # it counts in what a batch's size is taken from, and is only tried for
    src = (ROOT / "bzip2gpu_b200" / "csrc" / "decode.cu").read_text()
    held = src[src.index("size_t held() const"):]
    held = held[:held.index("return s;")]
    for name in ("jumps", "lutlen", "maps"):
        assert f"&{name}" in held
        assert f"reserve(w.{name}" not in src or name == "maps"
    assert "w.jumps.try_reserve" in src
