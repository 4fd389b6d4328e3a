"""CPU tests of what the compiler made of the kernels."""
import re


def tiled_forms():
    """{(bits, group, output mode, scales in shared memory): (bytes of spill stores, bytes of static shared memory)} of the tiled tcgen05 kernel, as ptxas
    reported them when it was built."""
    from strixite_b200 import build
    found = re.findall(r"Compiling entry function '\S*tiled_tc_kernelILi(\d)ELi(\d+)ELi(\d)ELb(\d)E\S*' for 'sm_100a'\n.*\n"
                       r"\s*\d+ bytes stack frame, (\d+) bytes spill stores.*\n.*?(?:, (\d+) bytes smem)?\n", build.ptxas_report("grouped_tc_tiled").read_text())
    assert len(found) == 54  # Q4, Q8 x three group sizes x (four output modes with and without shared-memory scales, and the up mix)
    return {tuple(f[:4]): (int(f[4]), int(f[5])) for f in found}


def test_tiled_kernel_keeps_to_its_registers(lib):
    """The 24 warps of the tiled tcgen05 kernel have 80 registers each and 28 to 60 KB of L1 between them.  Spilled registers take the lines in which
    the producers find their scales: 108 bytes a thread made the SwiGLU form 15 % slower.  Q8 with groups of 32 (four groups a step) has always spilled some."""
    over = {f: n for f, (n, _) in tiled_forms().items() if n > (60 if f[:2] == ("8", "32") and f[3] == "0" else 8)}
    assert not over, over


def test_tiled_kernel_fits_a_cta_s_shared_memory(lib):
    """227 KB of a CTA less the largest dynamic part, 128 KB of stages, 64 of ring slots and 32 of scales; the rest of the forms ask for less."""
    over = {f: n for f, (_, n) in tiled_forms().items() if not 0 < n <= (227 - 128 - 64 - 32) * 1024}
    assert not over, over
