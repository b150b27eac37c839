"""Every kernel that is launched with programmatic stream serialisation (pdl.cuh)
waits for the stream's earlier kernels: its body calls pdl_begin() or one of
fused.cuh's twiddle loads, which end in the wait."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "monofonic_gb300" / "csrc"


def bodies(text):
    """{name: body} of the kernels and of the z passes that some of them consist of."""
    out = {}
    for m in re.finditer(r"(?:__global__[^;{]*?\b(?=k_)|__device__[^;{]*?\b(?=z_rows))(\w+)\s*\([^;{]*?\)\s*\{", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out[m.group(1)] = text[m.end():end]
    return out


def test_overlapping_launches_wait():
    kernels, launched = {}, set()
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        kernels.update(bodies(text))
        launched |= set(re.findall(r"(?:launch_pdl|MFX_FF_PERSISTENT)\(\(?(k_\w+)", text))
    assert len(launched) >= 39 and launched <= set(kernels), launched - set(kernels)
    waits = re.compile(r"pdl_begin\(\)|load_tw(_steps)?<")
    parts = [k for k in kernels if not k.startswith("k_") and waits.search(kernels[k])]
    assert len(parts) == 2
    waits = re.compile("|".join([waits.pattern] + [p + "<" for p in parts]))
    assert not [k for k in sorted(launched) if not waits.search(kernels[k])]
