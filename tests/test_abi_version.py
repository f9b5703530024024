"""The ABI version's minor step counts the additions: a caller that needs the
whole-frame encode asks for 1.2 (no GPU needed)."""
import vp8a


def test_version_names_the_whole_frame_encode():
    lib = vp8a.load()
    assert hasattr(lib, "vp8a_encode_inter_frame")
    assert lib.vp8a_abi_version() == 1 << 16 | 2
