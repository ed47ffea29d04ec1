"""Every thread that calls the library pays for its thread-local storage: the launchers keep one
table of occupancy answers, not one for each kernel type."""
import struct


def test_thread_local_segment_is_small(cuda_lib):
    from nt2_gb300.build import LIB
    with open(LIB, "rb") as f:
        elf = f.read()
    assert elf[:5] == b"\x7fELF\x02"                     # 64-bit
    phoff, = struct.unpack_from("<Q", elf, 32)
    phentsize, phnum = struct.unpack_from("<HH", elf, 54)
    tls = 0
    for i in range(phnum):
        kind, _, _, _, _, _, memsz, _ = struct.unpack_from("<IIQQQQQQ", elf, phoff + i * phentsize)
        if kind == 7:                                      # PT_TLS
            tls += memsz
    assert 0 < tls <= 16384
