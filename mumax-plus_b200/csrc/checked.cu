// checked.cu -- the index-checked library in one translation unit (the record of
// the first bad index is one device variable).
#include "engine.cu"
#include "xpass.cu"
#include "xthree.cu"
#include "yz.cu"
#include "yzwarp.cu"
#include "yzlong.cu"
#include "yzthree.cu"
#include "thick.cu"
#include "pairs.cu"
