"""sphdem_status_copy refuses null pointers before touching the GPU."""


def test_null_pointers_are_refused():
    from warp_sph_gpt_gb300 import build

    build.build_cuda()
    from warp_sph_gpt_gb300 import _lib

    lib = _lib.load()
    for ctl, host in ((None, 16), (16, None), (None, None)):
        assert lib.sphdem_status_copy(ctl, host, None, None) == 2
        assert b"null pointer" in lib.sphdem_last_error()
