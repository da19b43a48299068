"""Rules that kernels launched while the kernel before them still runs have to keep, read off the sources: a breach shows on a GPU only
when the timing is bad."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "adafactor-8bit_b200", "csrc")


def sources():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                out[name] = re.sub(r"//[^\n]*", "", f.read())
    return out


def kernels_after_others():
    """name -> text of the kernels that launch_next launches (by name, or as `kernel`, a name given a line or two before)."""
    src = sources()
    names = set()
    for text in src.values():
        for m in re.finditer(r"launch_next\((\w+)", text):
            names.add(m.group(1))
        if "launch_next(kernel" in text:
            names.update(re.findall(r"auto kernel = (\w+)", text))
    names -= {"kernel", "void"}
    out = {}
    for text in src.values():
        for m in re.finditer(r"^(?:template[^\n]*\n)?__global__.*?^\}", text, re.S | re.M):
            name = re.search(r"(\w+)\s*\((?!\()(?:const|void|double|FullrankLaunch|ScaleLaunch|\w+ \*)", re.sub(r"__launch_bounds__\([^\n]*", "", m.group(0))).group(1)
            if name in names:
                out[name] = m.group(0)
    return names, out


def test_every_kernel_is_found():
    names, found = kernels_after_others()
    assert len(names) >= 20 and names == set(found)


def test_kernels_wait_before_they_run_on():
    for name, text in kernels_after_others()[1].items():
        assert "await_launches()" in text or "write_units<" in text, name


# what these kernels call lies in these files or is no memory access
_CALLED = ("factored.cuh", "fullrank_fast.cuh", "fullrank_generic.cuh", "fullrank_stat.cuh", "fullrank_api.cuh", "launch.cuh", "scale.cuh",
           "schedule.cuh", "tensormap.cuh", "write_units.cuh", "common.cuh")


def test_no_read_only_loads():
    """The memory may still be written when the kernel starts: no __ldg, no ld.global.nc, no const __restrict__ parameter."""
    src = sources()
    for name in _CALLED:
        assert not re.search(r"__ldg\(|ld\.global\.nc", src[name]), name
    for name, text in kernels_after_others()[1].items():
        assert not re.search(r"__ldg\(|ld\.global\.nc|const (?!CUtensorMap)\w+ \*__restrict__", text), name


def test_tables_with_tensor_maps_are_released():
    """An upload by a kernel whose table holds tensor maps ends with the release that the acquire of their readers belongs to."""
    src = sources()
    assert "fence.proxy.tensormap::generic.acquire" in src["tensormap.cuh"]
    kernel = re.search(r"upload_kernel\(.*?^\}", src["launch.cuh"], re.S | re.M).group(0)
    assert re.search(r"dev\[i\] = [^;]*;\s*if \(MAPS\) asm volatile\(\"fence\.proxy\.tensormap::generic\.release", kernel)
    calls = [c for text in src.values() for c in re.findall(r"upload_table[^;]*;", text) if "MAPS" not in c]
    assert len(calls) >= 8
    maps = [c for c in calls if "CUtensorMap" in c or "UmmaTask" in c]
    assert len(maps) == 2 and all(c.startswith("upload_table<true>") for c in maps)


def test_an_upload_clears_no_error_but_its_own():
    body = re.search(r"upload_table\(void \*dev.*?^\}", sources()["launch.cuh"], re.S | re.M).group(0)
    assert body.count("cudaGetLastError") == 1
    assert re.search(r"cudaPointerGetAttributes\(&a, host\) != cudaSuccess\) \{\s*cudaGetLastError\(\);", body)


def test_a_write_pass_that_gives_up_waits_for_its_copies():
    """What the warp that copies has requested may still write shared memory: bounded waits for the stages come before the last arrival,
    on which the other warps leave."""
    text = sources()["write_units.cuh"]
    leave = re.search(r"if \(id < 0 \|\| given_up\) \{.*?return;", text, re.S).group(0)
    assert re.search(r"if \(given_up\)\s*for [^;]*;[^;]*;[^;]*mbar_wait_bounded\(&sh\.full\[k % NS\], \(k / NS\) & 1u\);.*mbarrier\.arrive", leave, re.S)
