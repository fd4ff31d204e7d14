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


def functions(text):
    """(name, parameters, body) of every function definition at namespace level that runs on the device."""
    for m in re.finditer(r"__(?:global|device)__[^;{}()]*(?:\([^()]*(?:\([^()]*\)[^()]*)*\))?[^;{}()]*?\b(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, brace = text[m.end():i - 1], text.find("{", i)
        if brace < 0 or text[i:brace].strip():
            continue  # a declaration, or a variable
        depth, j = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), params, text[brace:j]


#: What device code that runs behind another kernel's launch may read as data that stay the same while it is there: the
#: inputs of the call, and what was finished before the call's first launch.  k_region_pairs is such a first launch.
CONSTANT = {
    "k_project": {"indices", "vertices"}, "k_project_deferred": {"indices", "vertices"},
    "k_region_pairs": {"cum", "order", "ranked", "n_dev"}, "owners_of_items": {"cum"}, "first_rank_above": {"cum"},
    "item_pair": {"order", "ranked"}, "k_fine_lists": {"tile_start"}, "k_distortion_loss": {"dist", "d"},
    "k_clear_flagged_rows": {"tet_flags"},
    "k_backward": {"ranges", "records", "jitter", "out_img", "dist_img", "hit_counts", "hit_ids", "hit_masks", "g_img", "g_dist",
                   "gd"},
}


def test_kernels_behind_others_do_not_read_what_those_write_as_constant_data():
    texts, seen = sources(), set()
    for name, text in texts.items():
        for fn, params, body in functions(text):
            if "after_previous();" not in body and name != "rm_binning.cu":
                continue
            seen.add(fn)
            allowed = CONSTANT.get(fn, set())
            constant = set(re.findall(r"const[\w\s]*\*\s*__restrict__\s+(\w+)", params))
            assert constant <= allowed, (fn, constant - allowed)
            for arg in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?(\w+)", body):
                assert arg in allowed | {"rcam"}, (fn, arg)
    behind = re.findall(r"rm_launch_behind\([^;]*?(k_\w+)", " ".join(texts.values()))
    assert {"k_rank_rects", "k_digit_hist", "k_fine_lists", "k_distortion_loss_mean"} <= set(behind)
    assert set(behind) <= seen and {"k_rank_pass", "k_region_pass", "k_backward", "k_project_deferred"} <= seen


def test_asynchronous_copies_are_ordered_for_the_compiler():
    """An asm statement with a "memory" clobber is a place that no access to memory moves across."""
    found = [s for text in sources().values() for s in re.findall(r'asm volatile\((?:"[^"]*"|[^";])*;', text)
             if "cp.async" in s or "griddepcontrol" in s]
    assert len(found) >= 6
    for statement in found:
        assert '"memory"' in statement, statement
