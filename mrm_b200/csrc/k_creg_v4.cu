// k_creg_v4.cu -- register column kernel of compiled shape 4 (launch.h kCreg).
#define CREG_V 4
#include "k_creg.inc"
