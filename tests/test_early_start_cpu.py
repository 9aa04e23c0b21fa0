"""What a kernel that starts before its predecessor has completed may read through the non-coherent path: weights, which the
predecessor does not write.  Everything else takes ordinary loads, which its dependency wait orders."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blackwell_b200", "csrc")
WEIGHTS = {"W", "w", "wrow", "c.w", "c.bias"}


def test_only_weights_are_read_through_the_non_coherent_path():
    text = {os.path.basename(p): open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))}
    ordinary = set(re.findall(r"(\w+)(?:<[^<>;]*>)?<<<", "".join(text.values())))   # kernels that never start early
    wrong, seen = [], 0
    for name, s in sorted(text.items()):
        early = "pdl_wait" in s or "launch_pdl" in s or name.endswith(".cuh")
        function = ""
        for i, line in enumerate(s.splitlines(), 1):
            start = re.match(r"(?:__global__.*?|__device__.*?)?(\w+)\((?!\d)", line) if re.match(r"\w", line) else None
            if start and not line.startswith(("template", "static_assert", "#")):
                named = re.findall(r"(\w+)\((?!\d)", re.sub(r"__launch_bounds__\([^)]*\)", "", line))
                function = named[0] if named else function
            for arg in re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()*\(*(?:static_cast<[^>]*>\()*([\w.]+)", re.sub(r"//.*", "", line)):
                seen += 1
                if early and function not in ordinary and arg not in WEIGHTS:
                    wrong.append((name, i, function, arg))
    assert seen > 5
    assert not wrong, wrong
