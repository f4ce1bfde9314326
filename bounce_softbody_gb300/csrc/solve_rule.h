// Which team solves a single body.
#pragma once

namespace b3g {

// CTAs of the one cluster that solves a small body, 0 for a body that takes the grid team: about two
// slices a CTA, up to eight on `widest` CTAs, the most (a power of two, at most 16) of which a cluster can
// be resident; 0: none can. Measured with the grid team / 8 / 4 / 2 slices a CTA, us a step:
// 378 vertices with three Newton iterations 823 / 723 / 657 / 628, 10^3 block 215 / 208 / 186 / 179, cloth of
// 3721 vertices 220 / 186 / 183 / 183.
inline int cluster_ctas(int nslices, int widest)
{
	int cl = 1;
	while (cl < widest && nslices > 2 * cl) cl *= 2;
	return cl <= widest && nslices <= 8 * cl ? cl : 0;
}

} // namespace b3g
