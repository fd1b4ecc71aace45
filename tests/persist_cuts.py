"""Cuts of a persistent launch ("unit,most,snap,split", RK_NPU_B200_PERSIST_CUT) and the problems they are tried on: every width
of an item in every kernel, runs of items that begin and end inside a channel tile, accumulators taken again by a later item, and K
in parts with every number of pieces a thread takes turns at.  test_host_rules.py checks that the cuts do that on a GPU of
74 CTA pairs, test_gpu_persist_items.py runs them."""
UNITS = range(32, 257, 32)
GRIDS = [f"{u},1,0,1" for u in UNITS]                                    # items of one width, the last of a channel tile cut
RUNS = [f"32,{most},{snap},1" for most in range(2, 9) for snap in (0, 2, 3)]
PARTS = [f"{u},1,0,{s}" for u in UNITS if u <= 160 for s in (2, 3, 4, 6, 8)]

# tokens, K, accumulator rows: 49 units of 32 tokens and 20 channel tiles (the last of them cut); K of five k-blocks
WHOLE = (1541, 640, 5000)
WHOLE_FFN = (1541, 640, 5056)                                            # features in groups of 32: 2528
# K of 33 k-blocks for few channel tiles
LONG = (165, 4200, 702)
LONG_FFN = (165, 4200, 704)
