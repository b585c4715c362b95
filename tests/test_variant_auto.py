"""Selecting the forward's tile variant by grid size is a value of its own of
sgb_set_stream_config (host-only: nothing is launched)."""


def test_automatic_forward_variant():
    from seistorch_gb300 import _native, tuning
    lib = _native.load()
    try:
        assert tuning.AUTO >= len(tuning.FWD_VARIANTS)
        assert lib.sgb_set_stream_config(0, tuning.AUTO, 0) != 0
        assert lib.sgb_set_stream_config(tuning.AUTO - 1, 0, 0) != 0
        assert lib.sgb_set_stream_config(0, 0, tuning.AUTO) != 0
    finally:
        assert lib.sgb_set_stream_config(tuning.AUTO, tuning.DEFAULT[1], 0) == 0
