"""Rules that every kernel launch of the library keeps, checked on the sources: a launch that fails, or a load that is not
ordered behind the kernel before, shows up on a GPU only by chance, if at all."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "radiance_meshes_b200", "csrc")


def sources():
    """{file name: text without comments} of the CUDA sources."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        out[os.path.basename(path)] = re.sub(r"//[^\n]*", "", text)
    return out


def test_every_launch_returns_its_own_error():
    """No kernel is launched past the checked helpers: an unchecked launch that fails leaves the next kernel to run on memory
    that nobody has written, and its error to whoever asks the runtime next."""
    launches = 0
    for name, text in sources().items():
        assert "<<<" not in text, name
        if name == "rm_common.cuh":  # where the helpers are
            continue
        for m in re.finditer(r"\brm_launch(_behind|_config)?\(", text):
            assert text[:m.start()].rstrip().endswith("RM_CUDA_CHECK("), (name, text[m.start():m.start() + 80])
            launches += 1
    assert launches >= 20
