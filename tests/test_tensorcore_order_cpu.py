"""The order of two tcgen05.mma of one thread is guaranteed when they have the
same accumulator and the same shape, so every instruction descriptor of the
complex update has to give one shape: descriptors of the source, compiled and
decoded on the host."""
import os
import re
import subprocess

SOURCE = os.path.join(os.path.dirname(__file__), "..", "capytaine_b200", "csrc", "tc_gemm.cu")


def test_instruction_descriptors_have_one_shape(tmp_path):
    text = open(SOURCE).read()
    sizes = re.findall(r"^constexpr int kT(?:M|N|Nc) = [^;]+;", text, re.M)
    function = re.search(r"^constexpr uint32_t idesc_tf32\(.*?^}", text, re.M | re.S).group(0)
    descriptors = re.findall(r"^constexpr uint32_t (kIdesc\w*) = [^;]+;", text, re.M)
    definitions = re.findall(r"^constexpr uint32_t kIdesc\w* = [^;]+;", text, re.M)
    assert len(descriptors) >= 2
    main = "#include <cstdint>\n#include <cstdio>\n" + "\n".join([*sizes, function, *definitions]) + "\nint main() {\n"
    main += "".join(f'  std::printf("%u\\n", {d});\n' for d in descriptors) + "}\n"
    (tmp_path / "d.cpp").write_text(main)
    subprocess.run(["g++", "-std=c++17", "-o", str(tmp_path / "d"), str(tmp_path / "d.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "d")], check=True, capture_output=True, text=True).stdout.split()
    # M / 16 in bits 24 to 28, N / 8 in bits 17 to 22
    shapes = {(16 * (int(v) >> 24 & 31), 8 * (int(v) >> 17 & 63)) for v in out}
    assert len(shapes) == 1, shapes
    # and no instruction takes its descriptor from elsewhere
    calls = re.findall(r"mma_tf32\(tacc[^;]*;", text)
    assert calls and all(any(re.search(rf"\b{d}\b", c) for d in descriptors) for c in calls)
